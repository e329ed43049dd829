// prefill_umma.cuh — prompt batches of K-quant matrices (Q4_K / Q5_K / Q6_K x Q8_K) on the 5th-generation tensor cores, BIT-EXACT with
// the reference's CPU arithmetic (the counterpart of ggml-cuda's mul_mat_q, cpp/ggml/src/ggml-cuda/mmq.cuh).
//
// What has to be reproduced (cpp/ggml/src/ggml-quants.c:6914-6977, 7487-7560, 8145-8220): per output element (row, token) and per
// 256-weight super-block b, the AVX2 code forms EIGHT 32-bit integers — lane m sums scale[g] * w * a over bytes 4m..4m+3 of every
// 32-byte group g — and runs acc[m] = fma(d_b, (float) isum[m], acc[m]) block after block (plus 4 / 1 chains of mins x bsums). The
// fp32 chains are ordered; the integers are not. So:
//   * lane m of a super-block is a K = 32 contraction (8 groups x 4 bytes) with the 6-bit / 8-bit sub-block scale folded INTO the
//     weight: w * scale <= 15*63 = 945 (Q4_K), 31*63 = 1953 (Q5_K) — fp16 integers (<= 2048). Q6_K's (q - 32) * scale, up to 4096, is the
//     sum of two fp16 numbers, (q & 15) * scale <= 1920 and 16 ((q >> 4) - 2) * scale, a multiple of 16. Activations are int8. Every
//     product is an integer below 2^19 and every partial sum of the 32 terms is below 2^24 (32 * 4096 * 127), so an fp16 MMA with fp32
//     accumulation returns EXACTLY (float) isum[m].
//   * the mins chains are contractions too: bsum (|.| <= 4064) = lo (0..63) + hi (multiple of 64), both fp16 integers, K = 16 = 8 groups x
//     (lo, hi); for Q4_K the four lanes l of the reference's _mm_madd_epi16 are four B columns per token.
//   * the chain step acc = fma(d, D, acc) runs on the drained accumulators, super-block after super-block.
//
// What bounds it: not the tensor cores but what surrounds them. Per output element and super-block 12 (Q4_K) accumulators leave tensor
// memory and take one fma each, and the 12 chains of an element live in registers, which caps the tile at 4096 elements per SM: 128 rows x
// 32 tokens, 192 of a thread's registers. Every weight is therefore expanded once per 32 tokens, and that expansion must not pass
// through shared memory (64 KB written and read again per super-block would take longer than the chains): the expanding warps
// write the A operand straight into tensor memory, from where tcgen05.mma takes it.
//
// Persistent, one CTA per SM, four warpgroups (setmaxnreg: 2 x 224 + 40 + 24 registers x 128 threads = the launch's 512 x 128):
//   warps 0-7   consume: one output row and 16 tokens per thread; tcgen05.ld as the MMAs of a half super-block complete (dfull), packed chain
//               fmas. Nothing of an element leaves its thread before its row is finished.
//   warps 8-11  expand: lane = row of a 32-row unit. Raw tile -> fp16 -> tcgen05.st, half a super-block (four lane-slices) at a time (afull).
//   warp 12     issues the bulk copies of raw tiles and activation records into a ring of stages (full / empty)
//   warps 13,14 issue the MMAs of half 0 / 1 once it is expanded and the consumers have drained its accumulators (dfree). Two issuers: one
//               thread issues an MMA in 44 clocks whatever its N, two keep the pipe at 23 each (N = 32).
// Expansion, tensor cores and chains of neighbouring super-blocks (and tiles) overlap; every buffer is a half super-block.
// Measured (B200, Q4_K, 28672 rows, k = 4096, 512 tokens): 1211 us with mma.sync (k_mma_batch), 492 us here (Q5_K 645, Q6_K 690, where the expansion is
// the longer side); issue slots 60 % busy, fp32 pipe 44 %, logic 35 %.
// Tensor memory (all 512 columns, so its base is 0): D main [0, 256) = slice m at 32 m | Q4_K, Q5_K: D mins [256, 384), A [384, 512) = slice m
//   at 16 m | Q6_K: A of slices 0-3 [384, 512), of slices 4-7 [256, 384), 16 columns per part.
#pragma once
#include "prefill_mma.cuh"

namespace b200 {

static constexpr int UM_NT = 32;               // tokens per tile
static constexpr int UM_ROWS = 128;            // rows per tile (four work units)
static constexpr int UM_THREADS = 512;
static constexpr int UM_MAX_STAGES = 6;
// activation record block of one (32-token chunk, super-block)
//   main  [8 lanes m][token/8][k-chunk j (4)][token%8][8 fp16]: chunk j = groups 2j, 2j+1 of lane-slice m, bytes in the order
//         (0, 2, 1, 3) (the order the expansion extracts nibble pairs in)
//   yd    f32[32]
//   m5    [token/8 (4)][k-chunk (2)][token%8][8 fp16]       kk = 2 g + part, all groups                      (Q5_K)
//   m4    [(32 l + token)/8 (16)][k-chunk (2)][.%8][8 fp16] the same, non-zero for g in {2l, 2l+1}           (Q4_K)
static constexpr int UM_REC_SLICE = UM_NT * 64;                // 2048
static constexpr int UM_OFF_YD = 8 * UM_REC_SLICE;             // 16384
static constexpr int UM_OFF_M5 = UM_OFF_YD + UM_NT * 4;        // 16512
static constexpr int UM_OFF_M4 = UM_OFF_M5 + UM_NT * 32;       // 17536
static constexpr int UM_REC_BYTES = UM_OFF_M4 + UM_NT * 128;   // 21632
__host__ __device__ __forceinline__ int um_rec_copy_bytes(int type) { return type == T_Q4_K ? UM_REC_BYTES : type == T_Q5_K ? UM_OFF_M4 : UM_OFF_M5; }
static constexpr int UM_A_MINS = UM_ROWS * 32;                 // mins operand in shared memory [16 row groups][2][8][16 B], two buffers
static constexpr int UM_OUT_STRIDE = 33;                       // finished values [warp (8)][token (16)][32 rows + 1]
static constexpr int UM_OUT_BYTES = 8 * 16 * UM_OUT_STRIDE * 4;
static constexpr int UM_FIXED_SMEM = 2 * UM_A_MINS + UM_OUT_BYTES;      // 25088: a multiple of 128
static constexpr uint32_t UM_COL_DM = 256, UM_COL_A = 384;
__host__ __device__ constexpr uint32_t um_a_col(int type, int half) { return type == T_Q6_K ? (half ? 256u : 384u) : UM_COL_A + 64u * (uint32_t) half; }

// ---- tcgen05 / TMEM wrappers (PTX ISA 8.6+, sm_100a) ----
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc_512(uint32_t smem_dst) {   // one whole warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_dst), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_512(uint32_t taddr) {    // the same warp
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(taddr), "r"(512u) : "memory");
}
// shared-memory matrix descriptor, K-major, no swizzle (cute::UMMA::SmemDescriptor): start >> 4 | LBO >> 4 << 16 | SBO >> 4 << 32 | version 1
__device__ __forceinline__ uint64_t um_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t) ((saddr >> 4) & 0x3fffu) | ((uint64_t) ((lbo >> 4) & 0x3fffu) << 16) | ((uint64_t) ((sbo >> 4) & 0x3fffu) << 32) | (1ull << 46);
}
// instruction descriptor (cute::UMMA::InstrDescriptor): D = F32, A = B = F16, both K-major, M = 128, N
__host__ __device__ constexpr uint32_t um_idesc(int n) { return (1u << 4) | ((uint32_t) (n >> 3) << 17) | ((uint32_t) (UM_ROWS >> 4) << 24); }
template <bool ACC> __device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t da, uint64_t db, uint32_t idesc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 :: "r"(d_tmem), "l"(da), "l"(db), "r"(idesc), "n"(ACC ? 1 : 0) : "memory");
}
// the A operand from tensor memory: lane = row, a 32-bit column = two consecutive k
template <bool ACC> __device__ __forceinline__ void umma_f16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t db, uint32_t idesc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 :: "r"(d_tmem), "r"(a_tmem), "l"(db), "r"(idesc), "n"(ACC ? 1 : 0) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :: "r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// (behind the wait: nothing that uses the registers is moved before it)
__device__ __forceinline__ void tmem_ld8_ready(uint32_t (&r)[8]) {
    asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]));
}
template <int N> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" :: "n"(N)); }
template <int N> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(N)); }

// k_quant_batch_mma, k_umma_batch's layout: token t's quantized image -> its rows of the chunk's record blocks
__device__ __forceinline__ void um_write_records(const ActSmem & A, int n256, uint8_t * rec, int t, int lane, int warp, int W) {
    const int chunk = t / UM_NT, j = t % UM_NT;
    for (int b = warp; b < n256; b += W) {
        uint8_t * r = rec + ((size_t) chunk * n256 + b) * UM_REC_BYTES;
        const int8_t * qb = A.q + (size_t) b * 256;
        {   // lane = (m, c): k-chunk c of lane-slice m = groups 2c, 2c+1, bytes 4m..4m+3 in the order (0, 2, 1, 3)
            const int m = lane >> 2, c = lane & 3;
            const uint32_t w0 = *reinterpret_cast<const uint32_t *>(qb + 64 * c + 4 * m);
            const uint32_t w1 = *reinterpret_cast<const uint32_t *>(qb + 64 * c + 32 + 4 * m);
            uint4 o;
            o.x = h2_ints(sbyte_of(w0, 0), sbyte_of(w0, 2)); o.y = h2_ints(sbyte_of(w0, 1), sbyte_of(w0, 3));
            o.z = h2_ints(sbyte_of(w1, 0), sbyte_of(w1, 2)); o.w = h2_ints(sbyte_of(w1, 1), sbyte_of(w1, 3));
            *reinterpret_cast<uint4 *>(r + m * UM_REC_SLICE + (j >> 3) * 512 + c * 128 + (j & 7) * 16) = o;
        }
        if (lane == 0) *reinterpret_cast<float *>(r + UM_OFF_YD + j * 4) = A.dx[b];
        if (lane < 10) {
            const int * bp = A.bp + (size_t) b * 8;
            const int ch = lane & 1;
            uint4 z = make_uint4(0u, 0u, 0u, 0u);
            if (lane < 8) {
                const int l = lane >> 1, n = UM_NT * l + j;
                if (ch == (l >> 1)) {
                    const int s0 = bp[2 * l], s1 = bp[2 * l + 1];
                    const int l0 = s0 & 63, l1 = s1 & 63;
                    const uint32_t p0 = h2_ints(l0, s0 - l0), p1 = h2_ints(l1, s1 - l1);
                    if (l & 1) { z.z = p0; z.w = p1; } else { z.x = p0; z.y = p1; }
                }
                *reinterpret_cast<uint4 *>(r + UM_OFF_M4 + (n >> 3) * 256 + ch * 128 + (n & 7) * 16) = z;
            } else {
                int s[4], lo[4];
#pragma unroll
                for (int i = 0; i < 4; i++) { s[i] = bp[4 * ch + i]; lo[i] = s[i] & 63; }
                z.x = h2_ints(lo[0], s[0] - lo[0]); z.y = h2_ints(lo[1], s[1] - lo[1]);
                z.z = h2_ints(lo[2], s[2] - lo[2]); z.w = h2_ints(lo[3], s[3] - lo[3]);
                *reinterpret_cast<uint4 *>(r + UM_OFF_M5 + (j >> 3) * 256 + ch * 128 + (j & 7) * 16) = z;
            }
        }
    }
}

static constexpr int UQ_BLOCK_REC = UM_NT * 64 + UM_NT * 4;    // records of one (32-token chunk, 32-weight block): [8-byte piece c (4)][token][8 fp16] | f32 d[32]
static constexpr int UQ_OFF_DX = UM_NT * 64;
// k_quant_batch_mma, layout 3: token t's Q8_0 image (natural order) -> its pieces of the chunk's record blocks
__device__ __forceinline__ void uq_write_records(const ActSmem & A, int n256, uint8_t * rec, int t, int lane, int warp, int W) {
    const int chunk = t / UM_NT, j = t % UM_NT, blk = lane >> 2, c = lane & 3;
    for (int b = warp; b < n256; b += W) {
        uint8_t * r = rec + (((size_t) chunk * n256 + b) * 8 + blk) * UQ_BLOCK_REC;
        const uint2 w = *reinterpret_cast<const uint2 *>(A.q + (size_t) b * 256 + 8 * lane);
        uint4 o;
        o.x = h2_ints(sbyte_of(w.x, 0), sbyte_of(w.x, 1)); o.y = h2_ints(sbyte_of(w.x, 2), sbyte_of(w.x, 3));
        o.z = h2_ints(sbyte_of(w.y, 0), sbyte_of(w.y, 1)); o.w = h2_ints(sbyte_of(w.y, 2), sbyte_of(w.y, 3));
        *reinterpret_cast<uint4 *>(r + c * (UM_NT * 16) + j * 16) = o;
        if (c == 0) *reinterpret_cast<float *>(r + UQ_OFF_DX + j * 4) = A.dx[b * 8 + blk];
    }
}

// k_quant_batch with the tensor-core record layouts (one CTA per token: the decode path's prologue, then the image is written out
// for k_mma_batch (layout 1), k_umma_batch (layout 2) or k_umma_batch_q80 (layout 3))
__global__ void __launch_bounds__(512) k_quant_batch_mma(const QuantBatchArgs a) {
    extern __shared__ __align__(16) uint8_t qb_smem[];
    __shared__ double red_smem[MV_MAX_WARPS];
    pdl_launch_dependents();
    const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, W = blockDim.x >> 5;
    const ActSmem A = act_smem_carve(qb_smem, a.k, a.act_q8_0);
    const bool norm = a.norm_w != nullptr;
    float ww[PRO_U][8] = {};
    if (norm) {
#pragma unroll
        for (int u = 0; u < PRO_U; u++) {
            const int b = warp + u * W;
            if (b < a.k / 256) ldg8(a.norm_w + b * 256 + lane * 8, ww[u]);
        }
    }
    pdl_wait();
    prologue_quantize<false, true>(a.X + (size_t) t * a.k, norm, a.eps, a.k, a.inv_k, a.act_q8_0, A, red_smem, ww, []() {}, W);
    __syncthreads();
    if (a.layout == 3) uq_write_records(A, a.k / 256, a.rec, t, lane, warp, W);
    else if (a.layout == 2) um_write_records(A, a.k / 256, a.rec, t, lane, warp, W);
    else mb_write_records(A, a.k / 256, a.rec, t, lane, warp, W);
}

// Half h (lane-slices 4h .. 4h+3) of one row's super-block -> the A operand in tensor memory (taddr: the half's first column in the warp's
// lane quarter). k order of a slice: k-chunk j = groups 2j, 2j+1, bytes (0, 2, 1, 3) of each, as the nibbles come out of a word. A field
// v in bits p.. of a half-word is made fp16 by its place: 0x6400 | v << p is 1024 + v 2^p, and one HFMA2 with (s / 2^p, -1024 s / 2^p) leaves v s,
// exactly (logic runs at half rate here, so shifts are what is saved).
template <int TYPE>
__device__ __forceinline__ void um_expand_half(const uint8_t * tile, int lane, int h, uint32_t taddr) {
    const uint8_t * sl = tile + lane * 16;
    if (TYPE == T_Q4_K || TYPE == T_Q5_K) {
        const uint4 sd = lds_u4(sl + 4096);
        uint4 H4 = make_uint4(0u, 0u, 0u, 0u);
        if (TYPE == T_Q5_K) H4 = lds_u4(sl + 4608 + h * 512);
#pragma unroll
        for (int s = 0; s < 2; s++) {                          // K = 16 step s: 64-weight groups j = 2s, 2s + 1
            const uint32_t scw = s ? (sd.z & 0x0f0f0f0fu) | ((sd.x >> 2) & 0x30303030u) : sd.x & 0x3f3f3f3fu;
            const uint4 Wa = lds_u4(sl + (4 * s + h) * 512), Wb = lds_u4(sl + (4 * s + 2 + h) * 512);
            __half2 sc[4], of[4];                              // low nibbles of j, j + 1: (s, -1024 s); high nibbles, in place: (s / 16, -64 s)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const __half2 v = __hsub2(bits_h2(__byte_perm(scw, 0x64646464u, 0x4040u + 0x0101u * i)), bits_h2(0x64006400u));
                sc[i] = (i & 1) ? __hmul2(v, bits_h2(0x2c002c00u)) : v;
                of[i] = __hmul2(v, (i & 1) ? bits_h2(0xd400d400u) : bits_h2(0xe400e400u));
            }
#pragma unroll
            for (int wi = 0; wi < 4; wi++) {
                uint32_t o[8];
#pragma unroll
                for (int jj = 0; jj < 2; jj++) {
                    const uint32_t W = word_of(jj ? Wb : Wa, wi), V = W >> 8;
                    uint32_t l02 = (W & 0x000f000fu) | 0x64006400u, h02 = (W & 0x00f000f0u) | 0x64006400u;
                    uint32_t l13 = (V & 0x000f000fu) | 0x64006400u, h13 = (V & 0x00f000f0u) | 0x64006400u;
                    if (TYPE == T_Q5_K) {   // qh bit 2j -> bit 4 of a low-nibble weight, bit 2j + 1 -> bit 8 of a high-nibble one in place
                        const uint32_t H = word_of(H4, wi);
                        const int b = 2 * (2 * s + jj);
                        const uint32_t x = b <= 4 ? H << (4 - b) : H >> (b - 4), y = H << (7 - b), z = H >> (4 + b), w = H >> (1 + b);
                        l02 |= x & 0x00100010u; h02 |= y & 0x01000100u;
                        l13 |= z & 0x00100010u; h13 |= w & 0x01000100u;
                    }
                    o[4 * jj]     = h2_bits(__hfma2(bits_h2(l02), sc[2 * jj], of[2 * jj]));
                    o[4 * jj + 1] = h2_bits(__hfma2(bits_h2(l13), sc[2 * jj], of[2 * jj]));
                    o[4 * jj + 2] = h2_bits(__hfma2(bits_h2(h02), sc[2 * jj + 1], of[2 * jj + 1]));
                    o[4 * jj + 3] = h2_bits(__hfma2(bits_h2(h13), sc[2 * jj + 1], of[2 * jj + 1]));
                }
                tmem_st8(taddr + 16 * wi + 8 * s, o);
            }
        }
    } else {   // Q6_K: slices 4h + wi are the 16-byte column mq = h; groups g = gl (low nibbles), gl + 2 (high) of half n -> k-chunk 2n + gh
        const uint4 scv = lds_u4(sl + 4096);
#pragma unroll
        for (int n = 0; n < 2; n++) {
            {   // (q & 15) * s: every nibble at bits 4-7, (1024 + 16 v) * (s / 16) - 64 s
                const uint4 q0 = lds_u4(sl + (4 * n + h) * 512), q1 = lds_u4(sl + (4 * n + 2 + h) * 512);
                __half2 sc[4], of[4];
#pragma unroll
                for (int g = 0; g < 4; g++) {                      // scale of group g: byte 8n + 2g + h
                    const uint32_t w = (g < 2 ? (n ? scv.z : scv.x) : (n ? scv.w : scv.y)) >> (8 * (2 * (g & 1) + h));
                    const __half2 v = __hsub2(bits_h2(__byte_perm(w ^ 0x80u, 0x64646464u, 0x4040u)), bits_h2(0x64806480u));
                    sc[g] = __hmul2(v, bits_h2(0x2c002c00u)); of[g] = __hmul2(v, bits_h2(0xd400d400u));
                }
#pragma unroll
                for (int wi = 0; wi < 4; wi++) {
                    uint32_t e[8];
#pragma unroll
                    for (int gl = 0; gl < 2; gl++) {
                        const uint32_t Q = word_of(gl ? q1 : q0, wi);
                        e[2 * gl]     = h2_bits(__hfma2(bits_h2(((Q << 4) & 0x00f000f0u) | 0x64006400u), sc[gl], of[gl]));
                        e[2 * gl + 1] = h2_bits(__hfma2(bits_h2(((Q >> 4) & 0x00f000f0u) | 0x64006400u), sc[gl], of[gl]));
                        e[2 * gl + 4] = h2_bits(__hfma2(bits_h2((Q & 0x00f000f0u) | 0x64006400u), sc[gl + 2], of[gl + 2]));
                        e[2 * gl + 5] = h2_bits(__hfma2(bits_h2(((Q >> 8) & 0x00f000f0u) | 0x64006400u), sc[gl + 2], of[gl + 2]));
                    }
                    tmem_st8(taddr + 32 * wi + 8 * n, e);
                }
            }
            {   // 16 (v - 2) * s, v = the two high bits: at bits 6-7, (1024 + 64 v) * (s / 4) - 288 s, or at bits 8-9, (1024 + 256 v) * (s / 16) - 96 s
                const uint4 qh = lds_u4(sl + 4608 + (2 * n + h) * 512);
                __half2 s4[4], o4[4], s16[4], o16[4];
#pragma unroll
                for (int g = 0; g < 4; g++) {
                    const uint32_t w = (g < 2 ? (n ? scv.z : scv.x) : (n ? scv.w : scv.y)) >> (8 * (2 * (g & 1) + h));
                    const __half2 v = __hsub2(bits_h2(__byte_perm(w ^ 0x80u, 0x64646464u, 0x4040u)), bits_h2(0x64806480u));
                    s4[g] = __hmul2(v, bits_h2(0x34003400u)); o4[g] = __hmul2(v, bits_h2(0xdc80dc80u));
                    s16[g] = __hmul2(v, bits_h2(0x2c002c00u)); o16[g] = __hmul2(v, bits_h2(0xd600d600u));
                }
#pragma unroll
                for (int wi = 0; wi < 4; wi++) {
                    const uint32_t Q = word_of(qh, wi), L6 = Q << 6, L2 = Q << 2, R4 = Q >> 4, R6 = Q >> 6;
                    uint32_t e[8];                               // k-chunk gh, group gl: g = gl + 2 gh; bytes (0, 2), (1, 3)
                    e[0] = h2_bits(__hfma2(bits_h2((L6 & 0x00c000c0u) | 0x64006400u), s4[0], o4[0]));
                    e[1] = h2_bits(__hfma2(bits_h2((Q & 0x03000300u) | 0x64006400u), s16[0], o16[0]));
                    e[2] = h2_bits(__hfma2(bits_h2((L6 & 0x03000300u) | 0x64006400u), s16[1], o16[1]));
                    e[3] = h2_bits(__hfma2(bits_h2((R4 & 0x00c000c0u) | 0x64006400u), s4[1], o4[1]));
                    e[4] = h2_bits(__hfma2(bits_h2((L2 & 0x00c000c0u) | 0x64006400u), s4[2], o4[2]));
                    e[5] = h2_bits(__hfma2(bits_h2((R4 & 0x03000300u) | 0x64006400u), s16[2], o16[2]));
                    e[6] = h2_bits(__hfma2(bits_h2((L2 & 0x03000300u) | 0x64006400u), s16[3], o16[3]));
                    e[7] = h2_bits(__hfma2(bits_h2((R6 & 0x03000300u) | 0x64006400u), s16[3], o16[3]));
                    tmem_st8(taddr + 32 * wi + 16 + 8 * n, e);
                }
            }
        }
    }
}
// mins operand of one row: kk = 2g + part <- m[g] for both parts
__device__ __forceinline__ void um_expand_mins(const uint8_t * tile, int lane, int row, uint8_t * As) {
    const uint4 sd = lds_u4(tile + lane * 16 + 4096);
    const uint32_t mw[2] = {sd.y & 0x3f3f3f3fu, ((sd.z >> 4) & 0x0f0f0f0fu) | ((sd.y >> 2) & 0x30303030u)};
#pragma unroll
    for (int c = 0; c < 2; c++) {
        uint32_t o[4];
#pragma unroll
        for (int i = 0; i < 4; i++) o[i] = h2_bits(__hsub2(bits_h2(__byte_perm(mw[c], 0x64646464u, 0x4040u + 0x0101u * i)), bits_h2(0x64006400u)));
        *reinterpret_cast<uint4 *>(As + (row >> 3) * 256 + c * 128 + (row & 7) * 16) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// a 128-row tile: up to four units of one segment
struct UmTile { int type, n_units, row0; uint32_t bytes; const uint8_t * tiles; };
__device__ __forceinline__ UmTile um_tile(const MatmulBatchArgs & a, int rt) {
    UmTile d;
    int row_base = 0, si = 0;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int nt = (a.seg[i].n_units + 3) / 4;
        if (si == i && i + 1 < a.n_seg && rt >= nt) { rt -= nt; row_base += a.seg[i].n_rows; si = i + 1; }
    }
    d.type = si == 0 ? a.seg[0].type : si == 1 ? a.seg[1].type : a.seg[2].type;
    d.bytes = (uint32_t) (si == 0 ? a.seg[0].tile_bytes : si == 1 ? a.seg[1].tile_bytes : a.seg[2].tile_bytes);
    const int units = si == 0 ? a.seg[0].n_units : si == 1 ? a.seg[1].n_units : a.seg[2].n_units;
    const uint8_t * p = si == 0 ? a.seg[0].p0 : si == 1 ? a.seg[1].p0 : a.seg[2].p0;
    d.n_units = min(4, units - 4 * rt);
    d.tiles = p + (size_t) (4 * rt) * a.tiles_unit * d.bytes;
    d.row0 = row_base + rt * UM_ROWS;
    return d;
}

// finished values out[token (16)][32 rows] of one unit -> the layer's epilogue (pb_epilogue's arithmetic, a warp at a time). A token's 32 rows are
// consecutive in memory; the gated unit takes two tokens' 16 row pairs at once.
__device__ __forceinline__ void um_epilogue(const MatmulBatchArgs & a, const float * out, int row0, int tok0, int lane) {
    const int nt = min(16, a.T - tok0), row = row0 + lane;
    if (a.epi == EPI_STORE) {
        for (int t = 0; t < nt; t++) a.out[(size_t) (tok0 + t) * a.out_stride + row] = out[t * UM_OUT_STRIDE + lane];
    } else if (a.epi == EPI_RESID) {
        float r[16];
#pragma unroll
        for (int t = 0; t < 16; t++) if (t < nt) r[t] = a.resid[(size_t) (tok0 + t) * a.resid_stride + row];
#pragma unroll
        for (int t = 0; t < 16; t++) if (t < nt) a.out[(size_t) (tok0 + t) * a.out_stride + row] = __fadd_rn(out[t * UM_OUT_STRIDE + lane], r[t]);
    } else if (a.epi == EPI_SILU) {
#pragma unroll 2
        for (int t = lane >> 4; t < nt; t += 2) {
            const float * o = out + t * UM_OUT_STRIDE + 2 * (lane & 15);
            a.out[(size_t) (tok0 + t) * a.out_stride + (row0 >> 1) + (lane & 15)] = __fmul_rn(silu_exact(o[0]), o[1]);
        }
    } else {   // EPI_QKV
#pragma unroll 4
        for (int t = 0; t < nt; t++) {
            const int pos = a.pos0 + tok0 + t;
            const float val = out[t * UM_OUT_STRIDE + lane];
            if (row < a.n_q + a.n_k) {
                const float oth = out[t * UM_OUT_STRIDE + (lane ^ 1)];
                const float v0 = (lane & 1) ? oth : val, v1 = (lane & 1) ? val : oth;
                const float2 cs = a.rope[(size_t) pos * (a.head_dim / 2) + (((row & ~1) & (a.head_dim - 1)) >> 1)];
                const float y = (lane & 1) ? __fadd_rn(__fmul_rn(v0, cs.y), __fmul_rn(v1, cs.x))
                                           : __fsub_rn(__fmul_rn(v0, cs.x), __fmul_rn(v1, cs.y));
                if (row < a.n_q) a.q_out[(size_t) (tok0 + t) * a.q_stride + row] = y;
                else a.k_cache[(size_t) pos * a.kv_dim + (row - a.n_q)] = __float2half_rn(y);
            } else {
                a.v_cache[(size_t) pos * a.kv_dim + (row - a.n_q - a.n_k)] = __float2half_rn(val);
            }
        }
    }
}

__global__ void __launch_bounds__(UM_THREADS, 1) k_umma_batch(const __grid_constant__ MatmulBatchArgs a) {
    extern __shared__ __align__(128) uint8_t um_smem[];
    __shared__ __align__(8) uint64_t bars[2 * UM_MAX_STAGES + 6];
    __shared__ uint32_t tmem_base_s;
    __shared__ int failed_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    volatile int * failed = &failed_s;
    uint8_t * amins = um_smem;
    float * outs = reinterpret_cast<float *>(um_smem + 2 * UM_A_MINS);
    uint8_t * stages = um_smem + UM_FIXED_SMEM;
    const int n_steps = a.tiles_unit, n_stages = a.mb_stages, n_tiles = a.um_row_tiles * a.um_tok_tiles;
    pdl_launch_dependents();
    const uint32_t b_full = smem_u32(&bars[0]), b_empty = b_full + 8 * UM_MAX_STAGES, b_afull = b_empty + 8 * UM_MAX_STAGES, b_dfull = b_afull + 16, b_dfree = b_dfull + 16;
    if (tid == 0) {
        failed_s = 0;
        for (int s = 0; s < n_stages; s++) { mbar_init(b_full + 8 * s, 1); mbar_init(b_empty + 8 * s, 8); }
        for (int h = 0; h < 2; h++) { mbar_init(b_afull + 8 * h, 4); mbar_init(b_dfull + 8 * h, 1); mbar_init(b_dfree + 8 * h, 8); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) tmem_alloc_512(smem_u32(&tmem_base_s));
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp != 12) pdl_wait();                 // (warp 12 waits behind its first copies)

    if (warp >= 12) {
        regs_dec<24>();
        if (warp == 12) {                       // bulk copies: super-block after super-block, over all tiles of the CTA
            uint32_t s = 0, par = 1;            // (a stage's first use waits for nothing)
            // one super-block of a tile -> stage s: the raw tiles and (a later call for those copied ahead) the records
            auto copy = [&](const UmTile & t, int tt, int step, uint32_t s, bool raw, bool recs) {
                const uint32_t rc = (uint32_t) um_rec_copy_bytes(t.type), dst = smem_u32(stages) + s * a.mb_stage_bytes, bar = b_full + 8 * s;
                if (raw) {
                    const uint8_t * src = t.tiles + (size_t) step * t.bytes;
                    mbar_expect_tx(bar, (uint32_t) t.n_units * t.bytes + rc);
                    for (int u = 0; u < t.n_units; u++) bulk_g2s(dst + u * a.mb_raw_stride, src + (size_t) u * n_steps * t.bytes, t.bytes, bar);
                }
                if (recs) bulk_g2s(dst + 4 * a.mb_raw_stride, a.rec + ((size_t) tt * n_steps + step) * UM_REC_BYTES, rc, bar);
            };
            const int early = min(n_stages, n_steps);
            for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
                const int rt = tile / a.um_tok_tiles, tt = tile - rt * a.um_tok_tiles;
                const UmTile t = um_tile(a, rt);
                const bool first = tile == (int) blockIdx.x;
                if (first) {                    // weights wait for nobody; the records are the previous kernel's
                    if (elect_one()) { for (int i = 0; i < early; i++) copy(t, tt, i, i, true, false); }
                    __syncwarp();
                    pdl_wait();
                }
#pragma unroll 1
                for (int step = 0; step < n_steps; step++) {
                    const bool ahead = first && step < early;
                    if (!ahead) um_wait(b_empty + 8 * s, par, failed, a.err);
                    if (elect_one() && !*failed) copy(t, tt, step, s, !ahead, true);
                    __syncwarp();
                    if (++s == (uint32_t) n_stages) { s = 0; par ^= 1u; }
                }
            }
            if (*failed) { for (int i = 0; i < 1000; i++) __nanosleep(1000); }      // copies nobody waited for end before the block does
        } else if (warp < 15) {                 // MMAs of half h
            const int h = warp - 13;
            uint32_t it = 0, s = 0;
            for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
                const int type = um_tile(a, tile / a.um_tok_tiles).type;
#pragma unroll 1
                for (int step = 0; step < n_steps; step++, it++) {
                    um_wait(b_dfree + 8 * h, (it & 1) ^ 1u, failed, a.err);          // (the first super-block waits for nothing)
                    um_wait(b_afull + 8 * h, it & 1, failed, a.err);
                    tc_fence_after();
                    const uint32_t r0 = smem_u32(stages) + s * a.mb_stage_bytes + 4 * a.mb_raw_stride, am = smem_u32(amins) + (it & 1) * UM_A_MINS;
                    const uint64_t b0 = um_desc(r0 + 4 * h * UM_REC_SLICE, 128, 512);
                    if (elect_one()) {
                        if (!*failed) {
                            if (type == T_Q6_K) {
#pragma unroll
                                for (int i = 0; i < 4; i++) {
                                    const uint32_t d = 32 * (4 * h + i), ac = um_a_col(T_Q6_K, h) + 32 * i;
                                    umma_f16_ta<false>(d, ac, b0 + (i * UM_REC_SLICE >> 4), um_idesc(UM_NT));
                                    umma_f16_ta<true>(d, ac + 8, b0 + ((i * UM_REC_SLICE + 256) >> 4), um_idesc(UM_NT));
                                    umma_f16_ta<true>(d, ac + 16, b0 + (i * UM_REC_SLICE >> 4), um_idesc(UM_NT));
                                    umma_f16_ta<true>(d, ac + 24, b0 + ((i * UM_REC_SLICE + 256) >> 4), um_idesc(UM_NT));
                                }
                            } else {
#pragma unroll
                                for (int i = 0; i < 4; i++) {
                                    const uint32_t d = 32 * (4 * h + i), ac = um_a_col(T_Q4_K, h) + 16 * i;
                                    umma_f16_ta<false>(d, ac, b0 + (i * UM_REC_SLICE >> 4), um_idesc(UM_NT));
                                    umma_f16_ta<true>(d, ac + 8, b0 + ((i * UM_REC_SLICE + 256) >> 4), um_idesc(UM_NT));
                                }
                                if (type == T_Q4_K) umma_f16<false>(UM_COL_DM + 64 * h, um_desc(am, 128, 256), um_desc(r0 + UM_OFF_M4 + 2048 * h, 128, 256), um_idesc(64));
                                else if (h == 1) umma_f16<false>(UM_COL_DM, um_desc(am, 128, 256), um_desc(r0 + UM_OFF_M5, 128, 256), um_idesc(UM_NT));
                            }
                        }
                        umma_commit(b_dfull + 8 * h);
                    }
                    __syncwarp();
                    if (++s == (uint32_t) n_stages) s = 0;
                }
            }
            if (*failed) { for (int i = 0; i < 1000; i++) __nanosleep(1000); }      // its MMAs end before tensor memory is given back
        }
    } else if (warp >= 8) {
        regs_dec<40>();
        const int q = warp & 3;
        const uint32_t tl = (uint32_t) (32 * q) << 16;
        uint32_t it = 0, st = 0, fpar = 0;
        int prev_type = -1;
        for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
            const UmTile t = um_tile(a, tile / a.um_tok_tiles);
            auto run = [&](auto tag) {
                constexpr int TYPE = decltype(tag)::value;
                if (prev_type >= 0 && prev_type != TYPE) {     // another layout of tensor memory: the last super-block's accumulators must be out of it
                    um_wait(b_dfree, (it - 1) & 1, failed, a.err);
                    um_wait(b_dfree + 8, (it - 1) & 1, failed, a.err);
                }
                prev_type = TYPE;
#pragma unroll 1
                for (int step = 0; step < n_steps; step++, it++) {
                    um_wait(b_full + 8 * st, fpar, failed, a.err);
                    const uint8_t * raw = stages + st * a.mb_stage_bytes + q * a.mb_raw_stride;
#pragma unroll 1
                    for (int h = 0; h < 2; h++) {
                        um_wait(b_dfull + 8 * h, (it & 1) ^ 1u, failed, a.err);     // the MMAs that read this half of A are done
                        tc_fence_after();
                        if (TYPE != T_Q6_K && h == 0) {
                            um_expand_mins(raw, lane, 32 * q + lane, amins + (it & 1) * UM_A_MINS);
                            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        }
                        um_expand_half<TYPE>(raw, lane, h, tl + um_a_col(TYPE, h));
                        tmem_st_wait();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(b_afull + 8 * h);
                    }
                    if (++st == (uint32_t) n_stages) { st = 0; fpar ^= 1u; }
                }
            };
            switch (t.type) {
                case T_Q4_K: run(TypeTag<T_Q4_K>{}); break;
                case T_Q5_K: run(TypeTag<T_Q5_K>{}); break;
                default:     run(TypeTag<T_Q6_K>{}); break;
            }
        }
    } else {
        regs_inc<224>();
        const int q = warp & 3, th = warp >> 2;                 // lane quarter (unit), token half
        const uint32_t tl = ((uint32_t) (32 * q) << 16) + 16 * th;
        float * out = outs + warp * (16 * UM_OUT_STRIDE);
        uint32_t it = 0, fpar = 0, st = 0;
        for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
            const int rt = tile / a.um_tok_tiles, tt = tile - rt * a.um_tok_tiles;
            const UmTile t = um_tile(a, rt);
            if (tt * UM_NT + 16 * th >= a.T) {                       // no tokens in this half: only the hand-overs
#pragma unroll 1
                for (int step = 0; step < n_steps; step++, it++) {
                    for (int h = 0; h < 2; h++) {
                        um_wait(b_dfull + 8 * h, it & 1, failed, a.err);
                        __syncwarp();                                // (a lane still at this phase would miss it, were the next one let in)
                        if (lane == 0) mbar_arrive(b_dfree + 8 * h);
                    }
                    if (lane == 0) mbar_arrive(b_empty + 8 * st);
                    if (++st == (uint32_t) n_stages) { st = 0; fpar ^= 1u; }
                }
                continue;
            }
            auto run = [&](auto tag) {
                constexpr int TYPE = decltype(tag)::value;
                constexpr int NM = TYPE == T_Q4_K ? 4 : TYPE == T_Q5_K ? 1 : 0;
                float2 acc[8 + NM][8];                           // [chain][token pair]
#pragma unroll
                for (int c = 0; c < 8 + NM; c++) {
#pragma unroll
                    for (int i = 0; i < 8; i++) acc[c][i] = make_float2(0.f, 0.f);
                }
#pragma unroll 1
                for (int step = 0; step < n_steps; step++, it++) {
                    const uint8_t * stage = stages + st * a.mb_stage_bytes;
                    um_wait(b_full + 8 * st, fpar, failed, a.err);             // (complete long since: the MMAs below read the same stage)
                    const float4 * yd = reinterpret_cast<const float4 *>(stage + 4 * a.mb_raw_stride + UM_OFF_YD) + 4 * th;
                    float dw, dm = 0.f;
                    if (TYPE == T_Q6_K) dw = __half2float(*reinterpret_cast<const __half *>(stage + q * a.mb_raw_stride + 6656 + lane * 2));
                    else {
                        const __half2 dmh = bits_h2(lds_u32(stage + q * a.mb_raw_stride + 4096 + lane * 16 + 12));
                        dw = __low2float(dmh); dm = -__high2float(dmh);
                    }
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        um_wait(b_dfull + 8 * h, it & 1, failed, a.err);
                        tc_fence_after();
                        // eight columns (tokens) at a time, the next eight on their way while these are added: i = (octet o, chain c of the half)
                        const int nc = TYPE == T_Q4_K ? 6 : TYPE == T_Q5_K && h == 1 ? 5 : 4;
                        uint32_t v[2][8];
                        auto col = [&](int i) -> uint32_t {
                            const int o = i / nc, c = i % nc;
                            return tl + 8 * o + (c < 4 ? 32 * (4 * h + c) : UM_COL_DM + (TYPE == T_Q4_K ? 64 * h + 32 * (c - 4) : 0));
                        };
                        tmem_ld8(col(0), v[0]);
                        float2 d[4];
#pragma unroll
                        for (int i = 0; i < 2 * nc; i++) {
                            const int o = i / nc, c = i % nc;
                            // d = y[i].d * fp16(x[i].d) (ggml-quants.c:6922), acc[m] = fma(d, (float) isum[m], acc[m]) (:6974);
                            // dmin = -y[i].d * fp16(x[i].dmin), acc_m lane l = fma(dmin, (float) (m[2l] bsum[2l] + m[2l+1] bsum[2l+1]), .) (:6931-6934)
                            if (c == 0 || c == 4) {
                                const float2 w = c == 0 ? make_float2(dw, dw) : make_float2(dm, dm);
                                const float4 y0 = yd[2 * o], y1 = yd[2 * o + 1];
                                d[0] = __fmul2_rn(make_float2(y0.x, y0.y), w); d[1] = __fmul2_rn(make_float2(y0.z, y0.w), w);
                                d[2] = __fmul2_rn(make_float2(y1.x, y1.y), w); d[3] = __fmul2_rn(make_float2(y1.z, y1.w), w);
                            }
                            tmem_ld_wait();
                            tmem_ld8_ready(v[i & 1]);
                            if (i + 1 < 2 * nc) tmem_ld8(col(i + 1), v[(i + 1) & 1]);
                            else {                               // everything of this half is in registers
                                tc_fence_before();
                                __syncwarp();
                                if (lane == 0) mbar_arrive(b_dfree + 8 * h);
                            }
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                float2 & x = acc[c < 4 ? 4 * h + c : TYPE == T_Q4_K ? 8 + 2 * h + (c - 4) : 8 + NM - 1][4 * o + k];
                                const float2 f = make_float2(__uint_as_float(v[i & 1][2 * k]), __uint_as_float(v[i & 1][2 * k + 1]));
                                if (TYPE == T_Q5_K && c == 4) {  // summs += dmin * (float) sum_g m[g] bsum[g] (:7516): two roundings
                                    x = make_float2(__fadd_rn(x.x, __fmul_rn(d[k].x, f.x)), __fadd_rn(x.y, __fmul_rn(d[k].y, f.y)));
                                } else x = __ffma2_rn(d[k], f, x);
                            }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(b_empty + 8 * st);
                    if (++st == (uint32_t) n_stages) { st = 0; fpar ^= 1u; }
                }
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    float c0[12], c1[12];
#pragma unroll
                    for (int c = 0; c < 8 + NM; c++) { c0[c] = acc[c][i].x; c1[c] = acc[c][i].y; }
                    out[(2 * i) * UM_OUT_STRIDE + lane] = finish_row<TYPE>(c0);
                    out[(2 * i + 1) * UM_OUT_STRIDE + lane] = finish_row<TYPE>(c1);
                }
            };
            switch (t.type) {
                case T_Q4_K: run(TypeTag<T_Q4_K>{}); break;
                case T_Q5_K: run(TypeTag<T_Q5_K>{}); break;
                default:     run(TypeTag<T_Q6_K>{}); break;
            }
            __syncwarp();
            if (q < t.n_units && !*failed) um_epilogue(a, out, t.row0 + 32 * q, tt * UM_NT + 16 * th, lane);
            __syncwarp();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) { tc_fence_after(); tmem_dealloc_512(tmem_base_s); }
}

}  // namespace b200
