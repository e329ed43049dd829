// prefill_umma_q80.cuh — prompt batches of Q8_0 matrices (Q8_0 x Q8_0) on the 5th-generation tensor cores, BIT-EXACT with the reference's CPU
// arithmetic (tinyBLAS_Q0_AVX, cpp/ggml/src/llamafile/sgemm.cpp; the counterpart of ggml-cuda's mul_mat_q, cpp/ggml/src/ggml-cuda/mmq.cuh).
//
// The reference keeps eight fp32 lanes per output: lane m sums the FOUR products of bytes 4m..4m+3 of a 32-weight block and runs
// acc[m] = fma(d_w d_a, (float) isum[m], acc[m]) block after block. Four-term sums are an MMA with a block-diagonal B: half a block is K = 16 = four
// lanes x four bytes, column (q, token) of B holds the token's bytes in rows 4q..4q+3 and zeros elsewhere, so one MMA of 128 rows x (4 lanes x 32
// tokens) leaves 128 x 128 lane sums as exact floats (|isum| <= 4 * 128 * 127 < 2^24, int8 values in fp16). A quarter of the tensor cores' products count, and
// that is enough: an output's eight chain steps of a block take the fp32 pipe twice as long as its two MMA columns take the tensor cores.
//
// What bounds it: the two consuming warps of a scheduler. Their chain steps, 64 packed fmas and 8 packed products per thread and block, take the fp32 pipe 288
// clocks; the accumulators' way out (a wait, one load of 64 columns, an arrival per half block) and the factors' are a serial chain in each warp that two warps
// hide in part only: 700 clocks a block in all, 500 with nothing else on the SM. Four fmas in a row share their factor: three 64-bit operands that are all new take
// a packed fma three clocks instead of two. Under ncu (gate|up of an 8B model, 512 tokens) 59 % of the issue slots, 27 % of the fp32 pipe and 17 % of the tensor pipe are busy. Twelve warps with 8 tokens each (24-token tiles) took as long; loads of 32 columns, one in flight while the other is added, spill.
// Measured (B200, 8 layers of an 8B model, 512 tokens): 32.0 ms of products with mma.sync (64 x 32 tiles, fragments through shared memory), 20.2 ms here.
//
// Persistent, one CTA per SM, four warpgroups (setmaxnreg: 2 x 224 + 40 + 24 registers x 128 threads = the launch's 512 x 128):
//   warps 0-7   consume: one output row and 16 tokens per thread; its eight chains per token are 128 registers. A half of a tile without tokens, or whose tokens another
//               block has (um_halves), is only handed over
//   warps 8-11  expand: lane = row of a 32-row unit, int8 -> fp16 -> tcgen05.st, two blocks at a time (pfull)
//   warp 12     bulk copies of raw tiles and activation records into a ring of stages of four blocks (full / empty)
//   warps 13,15 MMAs of half 0 / 1 of each block (dfull), once its operands are there and the consumers have drained the buffer (dfree). One issuer for both: 23.4 ms.
//   warp 14     spreads the activations over the block-diagonal operand: 8-byte pieces, the zeros around them are written once per launch (pfull)
// Tensor memory (all 512 columns, so its base is 0): D = three half blocks of 128 columns (64 th + 16 q + token % 16) | A [384, 512) = four slots of two blocks.
#pragma once
#include "prefill_umma.cuh"

namespace b200 {

static constexpr int UQ_STAGE_BLOCKS = 4;
static constexpr int UQ_RAW = UQ_STAGE_BLOCKS * 1088;          // one unit's tiles of a stage
static constexpr int UQ_STAGE = 4 * UQ_RAW + UQ_STAGE_BLOCKS * UQ_BLOCK_REC;    // 26112: a multiple of 128
static constexpr int UQ_STAGES = 4;
static constexpr int UQ_SLOTS = 4;                             // operand slots of two blocks
static constexpr int UQ_B_HALF = 128 * 32;                     // [column / 8 (16)][k-chunk (2)][column % 8][8 fp16]
static constexpr int UQ_B_SLOT = 4 * UQ_B_HALF;
static constexpr int UQ_SMEM = UQ_SLOTS * UQ_B_SLOT + UM_OUT_BYTES + UQ_STAGES * UQ_STAGE;
static constexpr uint32_t UQ_COL_A = 384;

__device__ __forceinline__ void tmem_ld64(uint32_t taddr, uint32_t (&r)[64]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x64.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, "
                 "%26, %27, %28, %29, %30, %31, %32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, %48, %49, "
                 "%50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%64];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
                   "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
                   "=r"(r[30]), "=r"(r[31]), "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
                   "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]), "=r"(r[48]), "=r"(r[49]),
                   "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]), "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]),
                   "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63]) : "r"(taddr) : "memory");
}
// (behind the wait: nothing that uses the registers is moved before it)
__device__ __forceinline__ void tmem_ld64_ready(uint32_t (&r)[64]) {
#pragma unroll
    for (int i = 0; i < 64; i += 8)
        asm volatile("" : "+r"(r[i]), "+r"(r[i + 1]), "+r"(r[i + 2]), "+r"(r[i + 3]), "+r"(r[i + 4]), "+r"(r[i + 5]), "+r"(r[i + 6]), "+r"(r[i + 7]));
}
// mbarrier arrive of one lane without a branch
__device__ __forceinline__ void mbar_arrive_if(uint32_t bar, uint32_t on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" :: "r"(bar), "r"(on) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 :: "r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
                    "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}

__global__ void __launch_bounds__(UM_THREADS, 1) k_umma_batch_q80(const __grid_constant__ MatmulBatchArgs a) {
    extern __shared__ __align__(128) uint8_t uq_smem[];
    __shared__ __align__(8) uint64_t bars[2 * UQ_STAGES + 2 * UQ_SLOTS + 6];
    __shared__ uint32_t tmem_base_s;
    __shared__ int failed_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    volatile int * failed = &failed_s;
    uint8_t * bop = uq_smem;
    float * outs = reinterpret_cast<float *>(uq_smem + UQ_SLOTS * UQ_B_SLOT);
    uint8_t * stages = uq_smem + UQ_SLOTS * UQ_B_SLOT + UM_OUT_BYTES;
    const int n_steps = a.tiles_unit / UQ_STAGE_BLOCKS, n_tiles = a.um_row_tiles * a.um_tok_tiles;
    const uint32_t b_full = smem_u32(&bars[0]), b_empty = b_full + 8 * UQ_STAGES, b_pfull = b_empty + 8 * UQ_STAGES, b_pempty = b_pfull + 8 * UQ_SLOTS;
    const uint32_t b_dfull = b_pempty + 8 * UQ_SLOTS, b_dfree = b_dfull + 24;
    // four blocks of a tile -> stage s
    auto copy = [&](const UmTile & t, int tt, int step, uint32_t s, bool raw, bool recs) {
        const uint32_t dst = smem_u32(stages) + s * UQ_STAGE, bar = b_full + 8 * s;
        if (raw) {
            const uint8_t * src = t.tiles + (size_t) step * UQ_RAW;
            mbar_expect_tx(bar, (uint32_t) t.n_units * UQ_RAW + UQ_STAGE_BLOCKS * UQ_BLOCK_REC);
            for (int u = 0; u < t.n_units; u++) bulk_g2s(dst + u * UQ_RAW, src + (size_t) u * a.tiles_unit * 1088, UQ_RAW, bar);
        }
        if (recs) bulk_g2s(dst + 4 * UQ_RAW, a.rec + ((size_t) (tt >> a.um_halves) * a.tiles_unit + step * UQ_STAGE_BLOCKS) * UQ_BLOCK_REC, UQ_STAGE_BLOCKS * UQ_BLOCK_REC, bar);
    };
    const int early = min(UQ_STAGES, n_steps);
    pdl_launch_dependents();
    if (tid == 12 * 32) {                       // the first tile's first weights are on their way while the operand is cleared; they wait for nobody
        failed_s = 0;
        for (int s = 0; s < UQ_STAGES; s++) { mbar_init(b_full + 8 * s, 1); mbar_init(b_empty + 8 * s, 13); }
        for (int s = 0; s < UQ_SLOTS; s++) { mbar_init(b_pfull + 8 * s, 5); mbar_init(b_pempty + 8 * s, 2); }
        for (int s = 0; s < 3; s++) { mbar_init(b_dfull + 8 * s, 1); mbar_init(b_dfree + 8 * s, 8); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        const int rt = blockIdx.x / a.um_tok_tiles;
        const UmTile t = um_tile(a, rt);
        for (int s = 0; s < early; s++) copy(t, blockIdx.x - rt * a.um_tok_tiles, s, s, true, false);
    }
    for (int i = tid; i < UQ_SLOTS * UQ_B_SLOT / 16; i += UM_THREADS) reinterpret_cast<uint4 *>(bop)[i] = make_uint4(0u, 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 0) tmem_alloc_512(smem_u32(&tmem_base_s));
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();

    if (warp >= 12) {
        regs_dec<24>();
        if (warp == 12) {                       // bulk copies: four blocks after four blocks, over all tiles of the CTA
            uint32_t s = 0, par = 1;            // (a stage's first use waits for nothing)
            for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
                const int rt = tile / a.um_tok_tiles, tt = tile - rt * a.um_tok_tiles;
                const UmTile t = um_tile(a, rt);
#pragma unroll 1
                for (int step = 0; step < n_steps; step++) {
                    const bool ahead = tile == (int) blockIdx.x && step < early;
                    if (!ahead) um_wait(b_empty + 8 * s, par, failed, a.err);
                    if (elect_one() && !*failed) copy(t, tt, step, s, !ahead, true);
                    __syncwarp();
                    if (++s == UQ_STAGES) { s = 0; par ^= 1u; }
                }
            }
            if (*failed) { for (int i = 0; i < 1000; i++) __nanosleep(1000); }      // copies nobody waited for end before the block does
        } else if (warp == 13 || warp == 15) {  // MMAs of half h of every block
            const uint32_t h = warp == 15;
            uint32_t p = 0, ppar = 0, d = h, dpar = 1;                               // (a buffer's first use waits for nothing)
            const uint64_t b0 = um_desc(smem_u32(bop) + h * UQ_B_HALF, 128, 256);
            for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
#pragma unroll 1
                for (int pair = 0; pair < 2 * n_steps; pair++) {
                    um_wait(b_pfull + 8 * p, ppar, failed, a.err);
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        um_wait(b_dfree + 8 * d, dpar, failed, a.err);
                        tc_fence_after();
                        if (elect_one()) {
                            if (!*failed) umma_f16_ta<false>(128 * d, UQ_COL_A + 32 * p + 16 * i + 8 * h, b0 + ((p * UQ_B_SLOT + 2 * i * UQ_B_HALF) >> 4), um_idesc(128));
                            umma_commit(b_dfull + 8 * d);
                            if (i == 1) umma_commit(b_pempty + 8 * p);
                        }
                        __syncwarp();
                        d += 2;
                        if (d >= 3) { d -= 3; dpar ^= 1u; }
                    }
                    if (++p == UQ_SLOTS) { p = 0; ppar ^= 1u; }
                }
            }
            if (*failed) { for (int i = 0; i < 1000; i++) __nanosleep(1000); }      // its MMAs end before tensor memory is given back
        } else if (warp == 14) {                // the block-diagonal operand: lane = token; piece (token, q) = column 64 (token / 16) + 16 q + token % 16, k = 4q..4q+3
            uint32_t s = 0, par = 0, p = 0, ppar = 1;
            const uint32_t col = (uint32_t) (lane >> 4) * (8 * 256) + (uint32_t) ((lane >> 3) & 1) * 256 + (uint32_t) (lane & 7) * 16;
            for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
#pragma unroll 1
                for (int pair = 0; pair < 2 * n_steps; pair++) {
                    if (!(pair & 1)) um_wait(b_full + 8 * s, par, failed, a.err);
                    um_wait(b_pempty + 8 * p, ppar, failed, a.err);
                    const uint8_t * r = stages + s * UQ_STAGE + 4 * UQ_RAW + (pair & 1) * (2 * UQ_BLOCK_REC) + lane * 16;
                    uint8_t * w = bop + p * UQ_B_SLOT + col;
#pragma unroll 1
                    for (int b = 0; b < 2; b++) {
#pragma unroll
                        for (int c = 0; c < 4; c++) {          // 8-byte pieces 2 (c & 1), 2 (c & 1) + 1 of half c >> 1
                            const uint4 v = *reinterpret_cast<const uint4 *>(r + b * UQ_BLOCK_REC + c * (UM_NT * 16));
                            uint8_t * o = w + (2 * b + (c >> 1)) * UQ_B_HALF + (c & 1) * (4 * 256 + 128);
                            *reinterpret_cast<uint2 *>(o) = make_uint2(v.x, v.y);
                            *reinterpret_cast<uint2 *>(o + 2 * 256 + 8) = make_uint2(v.z, v.w);
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) { mbar_arrive(b_pfull + 8 * p); if (pair & 1) mbar_arrive(b_empty + 8 * s); }
                    if (pair & 1) { if (++s == UQ_STAGES) { s = 0; par ^= 1u; } }
                    if (++p == UQ_SLOTS) { p = 0; ppar ^= 1u; }
                }
            }
        }
    } else if (warp >= 8) {
        regs_dec<40>();
        const int q = warp & 3;
        const uint32_t tl = ((uint32_t) (32 * q) << 16) + UQ_COL_A;
        const __half2 c1152 = bits_h2(0x64806480u);
        uint32_t s = 0, par = 0, p = 0, ppar = 1;
        for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
#pragma unroll 1
            for (int pair = 0; pair < 2 * n_steps; pair++) {
                if (!(pair & 1)) um_wait(b_full + 8 * s, par, failed, a.err);
                um_wait(b_pempty + 8 * p, ppar, failed, a.err);
                tc_fence_after();
                const uint8_t * raw = stages + s * UQ_STAGE + q * UQ_RAW + (pair & 1) * (2 * 1088) + lane * 16;
#pragma unroll
                for (int b = 0; b < 2; b++) {
                    uint32_t o[16];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const uint4 w = lds_u4(raw + b * 1088 + h * 512);
#pragma unroll
                        for (int i = 0; i < 4; i++) {          // b + 128 in 0..255; 0x6400 | v is 1024 + v
                            const uint32_t x = word_of(w, i) ^ 0x80808080u;
                            o[8 * h + 2 * i]     = h2_bits(__hsub2(bits_h2(__byte_perm(x, 0x64646464u, 0x4140u)), c1152));
                            o[8 * h + 2 * i + 1] = h2_bits(__hsub2(bits_h2(__byte_perm(x, 0x64646464u, 0x4342u)), c1152));
                        }
                    }
                    tmem_st16(tl + 32 * p + 16 * b, o);
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) { mbar_arrive(b_pfull + 8 * p); if (pair & 1) mbar_arrive(b_empty + 8 * s); }
                if (pair & 1) { if (++s == UQ_STAGES) { s = 0; par ^= 1u; } }
                if (++p == UQ_SLOTS) { p = 0; ppar ^= 1u; }
            }
        }
    } else {
        regs_inc<224>();
        const int q = warp & 3, th = warp >> 2;                 // lane quarter (unit), token half
        const uint32_t tl = ((uint32_t) (32 * q) << 16) + 64 * th;
        float * out = outs + warp * (16 * UM_OUT_STRIDE);
        uint32_t s = 0, par = 0, d = 0, dpar = 0;
        const uint32_t one = elect_one() ? 1u : 0u;
        for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
            const int rt = tile / a.um_tok_tiles, tt = tile - rt * a.um_tok_tiles;
            const UmTile t = um_tile(a, rt);
            const int tok0 = (tt >> a.um_halves) * UM_NT + 16 * th;
            if (tok0 >= a.T || (a.um_halves && (tt & 1) != th)) { // this half has no tokens, or another block has them: only the hand-overs
#pragma unroll 1
                for (int step = 0; step < n_steps; step++) {
#pragma unroll 1
                    for (int b = 0; b < 2 * UQ_STAGE_BLOCKS; b++) {
                        um_wait(b_dfull + 8 * d, dpar, failed, a.err);
                        __syncwarp();                            // (a lane still at this phase would miss it, were the next one let in)
                        mbar_arrive_if(b_dfree + 8 * d, one);
                        if (++d == 3) { d = 0; dpar ^= 1u; }
                    }
                    mbar_arrive_if(b_empty + 8 * s, one);
                    if (++s == UQ_STAGES) { s = 0; par ^= 1u; }
                }
                continue;
            }
            float2 acc[8][8];                                    // [lane m][token pair]
#pragma unroll
            for (int c = 0; c < 8; c++) {
#pragma unroll
                for (int i = 0; i < 8; i++) acc[c][i] = make_float2(0.f, 0.f);
            }
#pragma unroll 1
            for (int step = 0; step < n_steps; step++) {
                um_wait(b_full + 8 * s, par, failed, a.err);               // (complete long since: the MMAs read the same stage)
                const uint8_t * w = stages + s * UQ_STAGE + q * UQ_RAW + 1024 + lane * 2, * x = stages + s * UQ_STAGE + 4 * UQ_RAW + UQ_OFF_DX + 64 * th;
#pragma unroll 2
                for (int b = 0; b < UQ_STAGE_BLOCKS; b++) {
                    const float dw = __half2float(*reinterpret_cast<const __half *>(w + b * 1088));
                    float2 dd[8];                                // fp16(x.d) * fp16(y.d)
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float4 y = *reinterpret_cast<const float4 *>(x + b * UQ_BLOCK_REC + 16 * i);
                        dd[2 * i] = __fmul2_rn(make_float2(y.x, y.y), make_float2(dw, dw)); dd[2 * i + 1] = __fmul2_rn(make_float2(y.z, y.w), make_float2(dw, dw));
                    }
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        uint32_t v[64];
                        um_wait(b_dfull + 8 * d, dpar, failed, a.err);
                        tc_fence_after();
                        tmem_ld64(tl + 128 * d, v);
                        tmem_ld_wait();
                        tmem_ld64_ready(v);
                        tc_fence_before();
                        mbar_arrive_if(b_dfree + 8 * d, one);
                        if (++d == 3) { d = 0; dpar ^= 1u; }
#pragma unroll
                        for (int k = 0; k < 32; k++) {           // (four steps with the same factor: its registers are read once)
                            const int i = k >> 2, m = k & 3;
                            float2 & c = acc[4 * h + m][i];
                            c = __ffma2_rn(dd[i], make_float2(__uint_as_float(v[16 * m + 2 * i]), __uint_as_float(v[16 * m + 2 * i + 1])), c);
                        }
                    }
                }
                __syncwarp();
                mbar_arrive_if(b_empty + 8 * s, one);
                if (++s == UQ_STAGES) { s = 0; par ^= 1u; }
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                float c0[12], c1[12];
#pragma unroll
                for (int c = 0; c < 8; c++) { c0[c] = acc[c][i].x; c1[c] = acc[c][i].y; }
                out[(2 * i) * UM_OUT_STRIDE + lane] = finish_row<T_Q8_0>(c0);
                out[(2 * i + 1) * UM_OUT_STRIDE + lane] = finish_row<T_Q8_0>(c1);
            }
            __syncwarp();
            if (q < t.n_units && !*failed) um_epilogue(a, out, t.row0 + 32 * q, tok0, lane);
            __syncwarp();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) { tc_fence_after(); tmem_dealloc_512(tmem_base_s); }
}

}  // namespace b200
