// prefill.cuh — prompt batches (llama_decode with n_tokens > 1): the same arithmetic as the per-token kernels, with every
// weight tile fetched ONCE for a chunk of 64 tokens instead of once per token.
//
// The products run on the tensor cores (prefill_umma.cuh, prefill_mma.cuh); k_matmul_batch here is the dp4a kernel they are measured
// against, and takes what they do not: the reference's CPU result keeps EIGHT separate fp32 accumulators per output element (AVX2 lane m owns bytes
// 4m..4m+3 of every 32-byte group, cpp/ggml/src/ggml-quants.c:5361-5382, 6914-6977), and the 4-byte granularity is exactly dp4a's.
//
//   k_embed_batch   token_embd rows of T tokens -> X[T][n_embd]
//   k_quant_batch   per token: [RMSNorm * w] + Q8_K / Q8_0 quantization (prologue_quantize, the decode path's own code) into
//                   RECORDS in global memory, laid out [chunk of 64 tokens][256-weight block][token][record] so that the
//                   blocks of one K step of a whole chunk are one contiguous bulk copy
//   k_matmul_batch  CTA = (32-row unit, 64-token chunk), 16 warps x 4 tokens; per K step one TMA bulk copy of the weight
//                   tile(s) + one of the chunk's activation records into a 2-stage shared-memory ring (full / empty
//                   mbarriers); every warp computes tile_ints for its 4 tokens and advances 4 x 12 fp32 chains in
//                   registers; epilogues as in the per-token kernel (RoPE + KV-cache rows, +residual, SiLU*up, store)
#pragma once
#include "kernels.cuh"

namespace b200 {

static constexpr int PB_CHUNK = 64;            // tokens per CTA of the batched mat-mul
static constexpr int PB_WARPS = 16;
static constexpr int PB_TOK = PB_CHUNK / PB_WARPS;   // tokens per warp (chains in registers: 4 x 12)
static constexpr int PB_STAGES = 2;

// activation record of one token for one 256-weight block: q[256] | dx | bp[8] | as[64] (Q8_K; `as` only when a Q6_K
// matrix consumes the vector) or q[256] | dx[8] (Q8_0: eight 32-weight blocks)
__host__ __device__ __forceinline__ int pb_record_bytes(int act_q8_0, int with_as) {
    return act_q8_0 ? 256 + 32 : (with_as ? 256 + 16 + 32 + 256 : 256 + 16 + 32);   // dx padded to 16 bytes: bp / as stay 16-byte aligned
}

__global__ void k_embed_batch(int type, const uint8_t * __restrict__ rows, size_t row_bytes, int k, const int32_t * __restrict__ tokens,
                              float * __restrict__ X) {
    pdl_launch_dependents();
    const uint8_t * row = rows + (size_t) tokens[blockIdx.y] * row_bytes;
    float * out = X + (size_t) blockIdx.y * k;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k; i += gridDim.x * blockDim.x) out[i] = dequant_elem(type, row, i);
}

struct QuantBatchArgs {
    const float * X;          // [T][k]
    int k, T;
    const float * norm_w;     // nullptr: no norm
    float eps;
    double inv_k;
    int act_q8_0, with_as;
    uint8_t * rec;            // [ceil(T/64)][k/256][64][record]
    int layout;               // 0: records above (k_matmul_batch), 1: k_mma_batch blocks, 2: k_umma_batch blocks
};

// one CTA per token: the decode path's prologue (RMSNorm + quantization into shared memory), then the image is written out
// as records
__global__ void __launch_bounds__(512) k_quant_batch(const QuantBatchArgs a) {
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
    const int n256 = a.k / 256, rb = pb_record_bytes(a.act_q8_0, a.with_as);
    const int chunk = t / PB_CHUNK, j = t % PB_CHUNK;
    for (int b = warp; b < n256; b += W) {
        uint8_t * r = a.rec + (((size_t) chunk * n256 + b) * PB_CHUNK + j) * rb;
        *reinterpret_cast<uint2 *>(r + lane * 8) = *reinterpret_cast<const uint2 *>(A.q + (size_t) b * 256 + lane * 8);
        if (a.act_q8_0) {
            if (lane < 8) *reinterpret_cast<float *>(r + 256 + lane * 4) = A.dx[b * 8 + lane];
        } else {
            if (lane == 0) *reinterpret_cast<float *>(r + 256) = A.dx[b];
            if (lane < 8) *reinterpret_cast<int *>(r + 272 + lane * 4) = A.bp[(size_t) b * 8 + lane];
            if (a.with_as) *reinterpret_cast<int2 *>(r + 304 + lane * 8) = *reinterpret_cast<const int2 *>(A.as + (size_t) b * 64 + lane * 2);
        }
    }
}

// ------------------------------------------------------------------------------------------------------------
// attention of a prompt batch: k_attn_scores_batch writes the raw score rows, then
//   k_attn_softmax_rows  one warp per (token, head) row, in place: k_attn_softmax's arithmetic (max, ggml_v_expf, per-16
//                        _mm512_reduce_add_ps sums accumulated in double, * (float)(1/sum)), each row normalised ONCE
//   k_attn_softmax_block the same for long rows, a block per row
//   k_attn_pv_batch      tinyBLAS' 16 chains t = c, c+16, ... of every output, rows and dims tiled in registers.
//                        A token's probabilities end at its own padded length; beyond it p = 0 and fma(v, 0, acc) == acc,
//                        which is what the reference's masked (-inf -> 0) columns contribute (cpp/src/llama.cpp:14132-14200).
// ------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_attn_softmax_rows(const AttnArgs a, int nz) {
    const int lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5);
    pdl_launch_dependents();
    pdl_wait();
    if (row >= nz * a.n_head) return;
    const int z = row / a.n_head, h = row - z * a.n_head;
    const int n_pad = (a.n_kv_override + z + 31) / 32 * 32, n16 = n_pad / 16;
    float * S = a.S + (size_t) z * a.zs + (size_t) h * a.s_stride;
    float mx = -INFINITY;
    for (int gi = lane; gi < n16; gi += 32) {
        const float4 * r4 = reinterpret_cast<const float4 *>(S + 16 * gi);
#pragma unroll
        for (int q = 0; q < 4; q++) { const float4 v = r4[q]; mx = fmaxf(fmaxf(mx, fmaxf(v.x, v.y)), fmaxf(v.z, v.w)); }
    }
    mx = warp_max(mx);
    double part = 0.0;
    for (int gi = lane; gi < n16; gi += 32) {
        float4 * r4 = reinterpret_cast<float4 *>(S + 16 * gi);
        float4 t[2];
#pragma unroll 1
        for (int pq = 0; pq < 2; pq++) {                       // float4 pairs {0, 2} and {1, 3}: a[8+i] + a[i]
            float4 lo = r4[pq], hi = r4[pq + 2];
            lo.x = v_expf(__fsub_rn(lo.x, mx)); lo.y = v_expf(__fsub_rn(lo.y, mx)); lo.z = v_expf(__fsub_rn(lo.z, mx)); lo.w = v_expf(__fsub_rn(lo.w, mx));
            hi.x = v_expf(__fsub_rn(hi.x, mx)); hi.y = v_expf(__fsub_rn(hi.y, mx)); hi.z = v_expf(__fsub_rn(hi.z, mx)); hi.w = v_expf(__fsub_rn(hi.w, mx));
            r4[pq] = lo; r4[pq + 2] = hi;
            const float4 tt = make_float4(__fadd_rn(hi.x, lo.x), __fadd_rn(hi.y, lo.y), __fadd_rn(hi.z, lo.z), __fadd_rn(hi.w, lo.w));
            if (pq) t[1] = tt; else t[0] = tt;
        }
        const float u0 = __fadd_rn(t[1].x, t[0].x), u1 = __fadd_rn(t[1].y, t[0].y), u2 = __fadd_rn(t[1].z, t[0].z), u3 = __fadd_rn(t[1].w, t[0].w);
        part += (double) __fadd_rn(__fadd_rn(u0, u2), __fadd_rn(u1, u3));
    }
    const double sum = warp_sum_d(part);
    const float inv = (float) (1.0 / sum);
    for (int gi = lane; gi < n16; gi += 32) {
        float4 * r4 = reinterpret_cast<float4 *>(S + 16 * gi);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            float4 v = r4[q];
            v.x = __fmul_rn(v.x, inv); v.y = __fmul_rn(v.y, inv); v.z = __fmul_rn(v.z, inv); v.w = __fmul_rn(v.w, inv);
            r4[q] = v;
        }
    }
}

// The same row by a whole block: every thread keeps its groups of 16 scores in registers, so that a row crosses memory once in and once out. The
// sums of 16 meet in shared memory and one warp adds them in k_attn_softmax_rows' order, bit for bit. A warp per row reads a long row three times
// and writes it twice, mostly past the L1: 288 tokens x 32 heads x 6288 keys 119 us against 225.
static constexpr int SMX_THREADS = 256, SMX_MAX_G = 4;        // rows of up to 256 * 16 * 4 = 16384 scores
static constexpr int SMX_MIN_ROW = 2048;                      // shorter rows leave most of a block idle: 256 tokens x 32 heads, two layers, rows of 1256 985 us with a warp each
                                                              // and 993 here, of 2056 1258 and 1236, of 8256 3514 and 3418
template <int G>
__global__ void __launch_bounds__(SMX_THREADS) k_attn_softmax_block(const AttnArgs a, int nz) {
    __shared__ float wmax[SMX_THREADS / 32], gsum[G * SMX_THREADS];
    __shared__ float inv_s;
    const int tid = threadIdx.x, lane = tid & 31, row = blockIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    const int z = row / a.n_head, h = row - z * a.n_head;
    const int n_pad = (a.n_kv_override + z + 31) / 32 * 32, n16 = n_pad / 16;
    float * S = a.S + (size_t) z * a.zs + (size_t) h * a.s_stride;
    float4 v[G][4];
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < G; i++) {
        const int gi = tid + i * SMX_THREADS;
        if (gi < n16) {
            const float4 * r4 = reinterpret_cast<const float4 *>(S + 16 * gi);
#pragma unroll
            for (int q = 0; q < 4; q++) v[i][q] = r4[q];
        } else {
#pragma unroll
            for (int q = 0; q < 4; q++) v[i][q] = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        }
    }
#pragma unroll
    for (int i = 0; i < G; i++) {
#pragma unroll
        for (int q = 0; q < 4; q++) mx = fmaxf(fmaxf(mx, fmaxf(v[i][q].x, v[i][q].y)), fmaxf(v[i][q].z, v[i][q].w));
    }
    mx = warp_max(mx);
    if (lane == 0) wmax[tid >> 5] = mx;
    __syncthreads();
    mx = wmax[0];
#pragma unroll
    for (int w = 1; w < SMX_THREADS / 32; w++) mx = fmaxf(mx, wmax[w]);
#pragma unroll 1
    for (int i = 0; i < G; i++) {
        const int gi = tid + i * SMX_THREADS;
        if (gi >= n16) break;
#pragma unroll
        for (int j = 0; j < G; j++) if (j == i) {
            float4 t[2];
#pragma unroll
            for (int pq = 0; pq < 2; pq++) {                   // float4 pairs {0, 2} and {1, 3}: a[8+i] + a[i]
                float4 lo = v[j][pq], hi = v[j][pq + 2];
                lo.x = v_expf(__fsub_rn(lo.x, mx)); lo.y = v_expf(__fsub_rn(lo.y, mx)); lo.z = v_expf(__fsub_rn(lo.z, mx)); lo.w = v_expf(__fsub_rn(lo.w, mx));
                hi.x = v_expf(__fsub_rn(hi.x, mx)); hi.y = v_expf(__fsub_rn(hi.y, mx)); hi.z = v_expf(__fsub_rn(hi.z, mx)); hi.w = v_expf(__fsub_rn(hi.w, mx));
                v[j][pq] = lo; v[j][pq + 2] = hi;
                t[pq] = make_float4(__fadd_rn(hi.x, lo.x), __fadd_rn(hi.y, lo.y), __fadd_rn(hi.z, lo.z), __fadd_rn(hi.w, lo.w));
            }
            const float u0 = __fadd_rn(t[1].x, t[0].x), u1 = __fadd_rn(t[1].y, t[0].y), u2 = __fadd_rn(t[1].z, t[0].z), u3 = __fadd_rn(t[1].w, t[0].w);
            gsum[gi] = __fadd_rn(__fadd_rn(u0, u2), __fadd_rn(u1, u3));
        }
    }
    __syncthreads();
    if (tid < 32) {
        double part = 0.0;
        for (int gi = lane; gi < n16; gi += 32) part += (double) gsum[gi];
        const double sum = warp_sum_d(part);
        if (lane == 0) inv_s = (float) (1.0 / sum);
    }
    __syncthreads();
    const float inv = inv_s;
#pragma unroll
    for (int i = 0; i < G; i++) {
        const int gi = tid + i * SMX_THREADS;
        if (gi < n16) {
            float4 * r4 = reinterpret_cast<float4 *>(S + 16 * gi);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                float4 x = v[i][q];
                x.x = __fmul_rn(x.x, inv); x.y = __fmul_rn(x.y, inv); x.z = __fmul_rn(x.z, inv); x.w = __fmul_rn(x.w, inv);
                r4[q] = x;
            }
        }
    }
}

// packed fp32 pairs: each half is the IEEE operation of the scalar instruction (a packed multiply whose only use is a packed add is
// contracted by the compiler: products that are added are not formed with these). In place of float2 and its intrinsics, with which k_attn_pv_batch needs more
// than its 128 registers (8 bytes spilled; 120 registers here).
__device__ __forceinline__ uint64_t pair_of(float lo, float hi) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ float2 unpair(uint64_t p) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p)); return r; }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) { uint64_t r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }

// scores of a prompt batch: CTA = (KV head, 128 keys, tq <= 16 tokens), a thread = one key, whose 128 values sit in registers as packed pairs for all
// tq x GQA dot products. Each is ggml_vec_dot_f16 on q rounded to f16: 4 accumulators x 16 lanes over i in {0, 64}, (0+2)+(1+3),
// _mm512_reduce_add_ps (cpp/ggml/src/ggml.c:12345-12371) — the batch > 1 branch of k_attn_scores — in 96 packed instructions and 32 broadcast
// loads of q, with no exchange between lanes. Bound by those loads and the packed arithmetic together (ncu: shared-memory pipe 84 %, fp32 pipe 58 %). Four
// lanes per key with scalar arithmetic: 512 tokens x 32 heads x 6256 keys 2.08 ms, now 1.03 ms. A token's row ends at its own padded length
// (-inf from its n_kv to there).
static constexpr int SCB_TQ = 16, SCB_KEYS = 128;
template <int GQA>
__global__ void __launch_bounds__(SCB_KEYS, 3) k_attn_scores_batch(const AttnArgs a, int nz, int tq) {
    constexpr int HD = 128;
    extern __shared__ __align__(16) uint8_t scb_dyn[];
    float * qs = reinterpret_cast<float *>(scb_dyn);                          // [tq * GQA][HD]
    pdl_launch_dependents();
    pdl_wait();
    const int g = blockIdx.x, tile = blockIdx.y, z0 = blockIdx.z * tq, tid = threadIdx.x;
    const int ntok = min(tq, nz - z0);
    const int n_kv_last = a.n_kv_override + z0 + ntok - 1;
    if (tile * SCB_KEYS >= (n_kv_last + 31) / 32 * 32) return;
    const int t = tile * SCB_KEYS + tid;
    for (int i = tid; i < ntok * GQA * (HD / 4); i += SCB_KEYS) {
        const int tok = i / (GQA * (HD / 4)), rem = i - tok * (GQA * (HD / 4));
        const float4 v = *reinterpret_cast<const float4 *>(a.q + (size_t) (z0 + tok) * a.zq + (size_t) (g * GQA) * HD + 4 * rem);
        reinterpret_cast<float4 *>(qs)[i] = make_float4(__half2float(__float2half_rn(v.x)), __half2float(__float2half_rn(v.y)),     // src1 converted to
                                                        __half2float(__float2half_rn(v.z)), __half2float(__float2half_rn(v.w)));    // the vec_dot_type F16
    }
    uint64_t kp[HD / 2];
#pragma unroll
    for (int s = 0; s < HD / 8; s++) {
        uint4 kv = make_uint4(0u, 0u, 0u, 0u);
        if (t < n_kv_last) kv = *reinterpret_cast<const uint4 *>(a.k_cache + (size_t) t * a.kv_dim + g * HD + 8 * s);
        const uint32_t w[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
        for (int i = 0; i < 4; i++) { const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[i])); kp[4 * s + i] = pair_of(f.x, f.y); }
    }
    __syncthreads();
#pragma unroll 1
    for (int r = 0; r < ntok * GQA; r++) {
        const int tok = r / GQA, h = r - tok * GQA;
        const int n_kv = a.n_kv_override + z0 + tok;
        if (t >= (n_kv + 31) / 32 * 32) continue;                  // (a multiple of 32: warp-uniform)
        const ulonglong2 * q = reinterpret_cast<const ulonglong2 *>(qs + (size_t) r * HD);       // two pairs each
        uint64_t ch[8];
#pragma unroll
        for (int p = 0; p < 8; p += 2) {
            uint64_t x[4], y[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const ulonglong2 q0 = q[(16 * j + 2 * p) / 4], q1 = q[(64 + 16 * j + 2 * p) / 4];
                x[j] = fma2(kp[32 + 8 * j + p], q1.x, mul2(kp[8 * j + p], q0.x));
                y[j] = fma2(kp[32 + 8 * j + p + 1], q1.y, mul2(kp[8 * j + p + 1], q0.y));
            }
            ch[p] = add2(add2(x[0], x[2]), add2(x[1], x[3]));
            ch[p + 1] = add2(add2(y[0], y[2]), add2(y[1], y[3]));
        }
        uint64_t t3[4], t6[2];
#pragma unroll
        for (int i = 0; i < 4; i++) t3[i] = add2(ch[4 + i], ch[i]);
#pragma unroll
        for (int i = 0; i < 2; i++) t6[i] = add2(t3[2 + i], t3[i]);
        const float2 u = unpair(add2(t6[0], t6[1]));
        const float res = __fadd_rn(u.x, u.y);
        a.S[(size_t) (z0 + tok) * a.zs + (size_t) (g * GQA + h) * a.s_stride + t] = t < n_kv ? __fmul_rn(res, a.scale) : -INFINITY;
    }
}

// P.V of a prompt batch: CTA = (KV head, 8 (token, head) rows), all 128 dims, two CTAs per SM. A half-warp is one of tinyBLAS' 16 chains (positions
// c, c + 16, ...), a lane 8 rows x 8 dims: 32 packed fmas per position on one 16-byte load of V (f16, converted in registers) and two of p.
// Bound by the fp32 pipe, with the loads close behind. 512 tokens x 32 heads x 6256 keys: 0.88 ms (1.90 with a thread per chain and dim, a load of p per fma).
static constexpr int PVB_CHUNK = 64;           // positions staged at a time
static constexpr int PVB_STAGES = 3;
static constexpr int PVB_THREADS = 256;
static constexpr int PVB_ROWS = 8;             // (token, head) rows per CTA
static constexpr int PVB_PS = PVB_ROWS + 4;    // floats of p per position (16-byte rows, stores two-way conflicted)
static constexpr int PVB_V_BYTES = PVB_CHUNK * 128 * 2, PVB_BUF_BYTES = PVB_V_BYTES + PVB_CHUNK * PVB_PS * 4;
static constexpr int PVB_RED_BYTES = 16 * PVB_ROWS * 128 * 4;  // final exchange [16 chains][8 rows][128 dims]
static constexpr int PVB_SMEM = PVB_STAGES * PVB_BUF_BYTES > PVB_RED_BYTES ? PVB_STAGES * PVB_BUF_BYTES : PVB_RED_BYTES;
template <int GQA>
__global__ void __launch_bounds__(PVB_THREADS, 2) k_attn_pv_batch(const AttnArgs a, int nz) {
    constexpr int HD = 128, TQ = PVB_ROWS / GQA;
    extern __shared__ __align__(16) uint8_t pvb_dyn[];
    pdl_launch_dependents();
    pdl_wait();
    const int g = blockIdx.x, z0 = blockIdx.y * TQ, tid = threadIdx.x, c = tid >> 4, dg = tid & 15;     // dims 8 dg .. 8 dg + 7
    const int ntok = min(TQ, nz - z0);
    const int n_kv_last = a.n_kv_override + z0 + ntok - 1;     // cells attended by the CTA's last token
    const int n_max = (n_kv_last + 31) / 32 * 32, n_chunks = (n_max + PVB_CHUNK - 1) / PVB_CHUNK;
    // p: threads 0..127 = (row, four positions); beyond a row's padded length p = 0 and fma(v, 0, acc) == acc
    const int pr = tid & 7, pq = (tid >> 3) & 15;
    const int ptok = pr / GQA, ph = pr - ptok * GQA;
    const int p_end = ptok < ntok ? (a.n_kv_override + z0 + ptok + 31) / 32 * 32 : 0;
    const float * prow = a.S + (size_t) (z0 + (ptok < ntok ? ptok : 0)) * a.zs + (size_t) (g * GQA + ph) * a.s_stride;
    float4 sp = make_float4(0.f, 0.f, 0.f, 0.f);
    auto load_v = [&](int ck) {                                 // V rows: 4 x 16 bytes a thread; rows beyond the last cell are zero
        if (ck < n_chunks) {
            uint8_t * base = pvb_dyn + (ck % PVB_STAGES) * PVB_BUF_BYTES;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int r = (tid >> 4) + 16 * i, t = ck * PVB_CHUNK + r;
                uint8_t * dst = base + r * (HD * 2) + dg * 16;
                if (t < n_kv_last) cp_async16(dst, a.v_cache + (size_t) t * a.kv_dim + g * HD + 8 * dg);
                else *reinterpret_cast<uint4 *>(dst) = make_uint4(0u, 0u, 0u, 0u);
            }
        }
        cp_async_commit();
    };
    auto load_p = [&](int ck) {
        const int t = ck * PVB_CHUNK + 4 * pq;
        sp = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tid < 128 && ck < n_chunks && t < p_end) sp = *reinterpret_cast<const float4 *>(prow + t);
    };
    auto stash_p = [&](int ck) {
        if (tid < 128 && ck < n_chunks) {
            float * pp = reinterpret_cast<float *>(pvb_dyn + (ck % PVB_STAGES) * PVB_BUF_BYTES + PVB_V_BYTES) + (4 * pq) * PVB_PS + pr;
            pp[0] = sp.x; pp[PVB_PS] = sp.y; pp[2 * PVB_PS] = sp.z; pp[3 * PVB_PS] = sp.w;
        }
    };
    uint64_t acc[PVB_ROWS][4];                                  // [row][dim pair]
#pragma unroll
    for (int r = 0; r < PVB_ROWS; r++) {
#pragma unroll
        for (int d = 0; d < 4; d++) acc[r][d] = 0ull;
    }
    load_p(0);
    load_v(0); load_v(1);
    stash_p(0);
    load_p(1);
#pragma unroll 1
    for (int ck = 0; ck < n_chunks; ck++) {
        cp_async_wait<PVB_STAGES - 2>();
        __syncthreads();                                        // chunk ck is complete, the buffer of ck - 1 is free
        load_v(ck + 2);
        stash_p(ck + 1);
        load_p(ck + 2);
        const uint8_t * base = pvb_dyn + (ck % PVB_STAGES) * PVB_BUF_BYTES;
#pragma unroll
        for (int s = 0; s < PVB_CHUNK / 16; s++) {
            const int tt = 16 * s + c;
            const uint4 vw = *reinterpret_cast<const uint4 *>(base + tt * (HD * 2) + dg * 16);
            const float4 * pp = reinterpret_cast<const float4 *>(base + PVB_V_BYTES + tt * (PVB_PS * 4));
            const float4 p0 = pp[0], p1 = pp[1];
            const uint32_t w[4] = {vw.x, vw.y, vw.z, vw.w};
            uint64_t v[4];
#pragma unroll
            for (int d = 0; d < 4; d++) { const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[d])); v[d] = pair_of(f.x, f.y); }
            const float p[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
#pragma unroll
            for (int r = 0; r < PVB_ROWS; r++) {
                const uint64_t p2 = pair_of(p[r], p[r]);
#pragma unroll
                for (int d = 0; d < 4; d++) acc[r][d] = fma2(v[d], p2, acc[r][d]);
            }
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    float * red = reinterpret_cast<float *>(pvb_dyn);
#pragma unroll
    for (int r = 0; r < PVB_ROWS; r++) {
        const float2 x0 = unpair(acc[r][0]), x1 = unpair(acc[r][1]), x2 = unpair(acc[r][2]), x3 = unpair(acc[r][3]);
        float4 * dst = reinterpret_cast<float4 *>(red + (size_t) (c * PVB_ROWS + r) * HD + 8 * dg);
        dst[0] = make_float4(x0.x, x0.y, x1.x, x1.y); dst[1] = make_float4(x2.x, x2.y, x3.x, x3.y);
    }
    __syncthreads();
    for (int i = tid; i < PVB_ROWS * HD; i += PVB_THREADS) {
        const int r = i / HD, d = i % HD, tok = r / GQA, h = r - tok * GQA;
        if (tok < ntok) {
            float t3[8], t6[4];                                   // _mm512_reduce_add_ps over the 16 chains
#pragma unroll
            for (int j = 0; j < 8; j++) t3[j] = __fadd_rn(red[(size_t) ((8 + j) * PVB_ROWS + r) * HD + d], red[(size_t) (j * PVB_ROWS + r) * HD + d]);
#pragma unroll
            for (int j = 0; j < 4; j++) t6[j] = __fadd_rn(t3[4 + j], t3[j]);
            a.out[(size_t) (z0 + tok) * a.zq + (size_t) (g * GQA + h) * HD + d] = __fadd_rn(__fadd_rn(t6[0], t6[2]), __fadd_rn(t6[1], t6[3]));
        }
    }
}

struct MatmulBatchArgs {
    TMat seg[3];
    int n_seg, n_units, k, tiles_unit;
    int act_q8_0, with_as;
    const uint8_t * rec;      // activation records (k_quant_batch)
    int T;
    int epi;
    float * out; int out_stride;          // [T][out_stride]
    const float * resid; int resid_stride;
    // EPI_QKV
    float * q_out; int q_stride;
    __half * k_cache; __half * v_cache;
    int n_q, n_k, head_dim, kv_dim;
    const float2 * rope;
    int pos0;                 // position (== KV cell) of token 0 of the batch
    // k_mma_batch (prefill_mma.cuh): shared-memory layout chosen on the host
    uint32_t mb_a_bytes, mb_raw_stride, mb_stage_bytes, mb_rec_copy;
    int mb_stages;
    int um_row_tiles, um_tok_tiles;       // k_umma_batch: 128-row tiles (of every segment by itself), 32-token tiles
    int um_halves;                        // k_umma_batch_q80: 1: um_tok_tiles counts halves of 16 tokens
    int * err;                            // raised by a kernel whose bounded wait ran out
};

// resolve a unit against the segments (same rule as describe_unit)
__device__ __forceinline__ UnitDesc pb_describe_unit(const MatmulBatchArgs & a, int unit) {
    int si = 0, u = unit, row_base = 0;
    if (a.n_seg > 1 && u >= a.seg[0].n_units) { u -= a.seg[0].n_units; row_base += a.seg[0].n_rows; si = 1;
        if (a.n_seg > 2 && u >= a.seg[1].n_units) { u -= a.seg[1].n_units; row_base += a.seg[1].n_rows; si = 2; } }
    UnitDesc d;
    d.type  = si == 0 ? a.seg[0].type : (si == 1 ? a.seg[1].type : a.seg[2].type);
    d.bytes = (uint32_t) (si == 0 ? a.seg[0].tile_bytes : (si == 1 ? a.seg[1].tile_bytes : a.seg[2].tile_bytes));
    const uint8_t * base = si == 0 ? a.seg[0].p0 : (si == 1 ? a.seg[1].p0 : a.seg[2].p0);
    d.tiles = base + (size_t) u * a.tiles_unit * d.bytes;
    d.row0  = row_base + u * 32;
    return d;
}

// the row's epilogue for token t (matvec_epilogue with per-token buffers)
__device__ __forceinline__ void pb_epilogue(const MatmulBatchArgs & a, float val, int row, int lane, int t) {
    const float oth = __shfl_xor_sync(0xffffffffu, val, 1);    // partner row (2i <-> 2i+1)
    if (t >= a.T) return;
    if (a.epi == EPI_STORE) {
        a.out[(size_t) t * a.out_stride + row] = val;
    } else if (a.epi == EPI_RESID) {
        a.out[(size_t) t * a.out_stride + row] = __fadd_rn(val, a.resid[(size_t) t * a.resid_stride + row]);
    } else if (a.epi == EPI_SILU) {
        if ((lane & 1) == 0) a.out[(size_t) t * a.out_stride + (row >> 1)] = __fmul_rn(silu_exact(val), oth);
    } else {  // EPI_QKV
        const int pos = a.pos0 + t;
        const float v0 = (lane & 1) ? oth : val, v1 = (lane & 1) ? val : oth;
        if (row < a.n_q + a.n_k) {
            const float2 cs = a.rope[(size_t) pos * (a.head_dim / 2) + (((row & ~1) & (a.head_dim - 1)) >> 1)];
            const float y = (lane & 1) ? __fadd_rn(__fmul_rn(v0, cs.y), __fmul_rn(v1, cs.x))
                                       : __fsub_rn(__fmul_rn(v0, cs.x), __fmul_rn(v1, cs.y));
            if (row < a.n_q) a.q_out[(size_t) t * a.q_stride + row] = y;
            else a.k_cache[(size_t) pos * a.kv_dim + (row - a.n_q)] = __float2half_rn(y);
        } else {
            a.v_cache[(size_t) pos * a.kv_dim + (row - a.n_q - a.n_k)] = __float2half_rn(val);
        }
    }
}

// shared memory of a stage: weight tiles of the step (8 consecutive 32-weight tiles for Q8_0, one tile otherwise) | records
__host__ __device__ __forceinline__ int pb_step_tiles(int act_q8_0) { return act_q8_0 ? 8 : 1; }
__host__ __device__ __forceinline__ size_t pb_stage_bytes(int max_tile_bytes, int act_q8_0, int with_as) {
    const size_t w = ((size_t) max_tile_bytes * pb_step_tiles(act_q8_0) + 127) / 128 * 128;
    return w + (size_t) PB_CHUNK * pb_record_bytes(act_q8_0, with_as);
}

__global__ void __launch_bounds__(PB_WARPS * 32, 1) k_matmul_batch(const __grid_constant__ MatmulBatchArgs a, int max_tile_bytes) {
    extern __shared__ __align__(128) uint8_t pb_smem[];
    __shared__ __align__(8) uint64_t bars[2 * PB_STAGES];      // full[stage], empty[stage]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chunk = blockIdx.x, unit = blockIdx.y;
    pdl_launch_dependents();
    pdl_wait();
    const int rb = pb_record_bytes(a.act_q8_0, a.with_as), st_tiles = pb_step_tiles(a.act_q8_0);
    const size_t w_bytes = ((size_t) max_tile_bytes * st_tiles + 127) / 128 * 128;
    const size_t stage_bytes = w_bytes + (size_t) PB_CHUNK * rb;
    const int n_steps = a.tiles_unit / st_tiles;                // K steps: 256 weights each
    const UnitDesc ud = pb_describe_unit(a, unit);
    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[PB_STAGES]);
    if (tid == 0) {
        for (int s = 0; s < PB_STAGES; s++) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, PB_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    const uint8_t * rec_chunk = a.rec + (size_t) chunk * (a.k / 256) * PB_CHUNK * rb;
    auto issue = [&](int step) {                               // thread 0: weights + the chunk's records of K step `step`
        const int s = step % PB_STAGES;
        const uint32_t dst = smem_u32(pb_smem + (size_t) s * stage_bytes);
        const uint32_t wb = ud.bytes * (uint32_t) st_tiles, ab = (uint32_t) (PB_CHUNK * rb);
        mbar_expect_tx(full0 + 8 * s, wb + ab);
        bulk_g2s(dst, ud.tiles + (size_t) step * wb, wb, full0 + 8 * s);
        bulk_g2s(dst + (uint32_t) w_bytes, rec_chunk + (size_t) step * PB_CHUNK * rb, ab, full0 + 8 * s);
    };
    if (tid == 0) { for (int s = 0; s < PB_STAGES && s < n_steps; s++) issue(s); }

    auto body = [&](auto tag) {
        constexpr int TYPE = decltype(tag)::value;
        float acc[PB_TOK][12];
#pragma unroll
        for (int j = 0; j < PB_TOK; j++) {
#pragma unroll
            for (int c = 0; c < 12; c++) acc[j][c] = 0.f;
        }
        for (int step = 0; step < n_steps; step++) {
            const int s = step % PB_STAGES;
            const uint32_t par = (uint32_t) ((step / PB_STAGES) & 1);
            mbar_wait(full0 + 8 * s, par);
            const uint8_t * stage = pb_smem + (size_t) s * stage_bytes;
            if (TYPE == T_Q8_0) {
                // eight 32-weight blocks per step; a block's weights are read once for the warp's four tokens. The lane sums
                // come out of dp4a already as floats: the accumulator input 0x4B400000 is the bit pattern of 1.5 * 2^23, and
                // adding an integer |v| < 2^22 to it gives the bit pattern of 12582912.0 + v — one exact FADD instead of an
                // I2F on the quarter-rate conversion pipe (|v| <= 4 * 127 * 127)
#pragma unroll 1
                for (int tt = 0; tt < 8; tt++) {
                    const uint8_t * tile = stage + (size_t) tt * ud.bytes, * sl = tile + lane * 16;
                    const uint4 w0 = lds_u4(sl), w1 = lds_u4(sl + 512);
                    const float dw = __half2float(*reinterpret_cast<const __half *>(tile + 1024 + lane * 2));
#pragma unroll
                    for (int j = 0; j < PB_TOK; j++) {
                        const uint8_t * r = stage + w_bytes + (size_t) (warp * PB_TOK + j) * rb;
                        const int4 a0 = *reinterpret_cast<const int4 *>(r + tt * 32), a1 = *reinterpret_cast<const int4 *>(r + tt * 32 + 16);
                        const float d = __fmul_rn(dw, *reinterpret_cast<const float *>(r + 256 + tt * 4));      // fp16(x.d) * fp16(y.d)
#pragma unroll
                        for (int wi = 0; wi < 4; wi++) {
                            const float f0 = __fsub_rn(__int_as_float(__dp4a((int) word_of(w0, wi), word_of(a0, wi), 0x4B400000)), 12582912.f);
                            const float f1 = __fsub_rn(__int_as_float(__dp4a((int) word_of(w1, wi), word_of(a1, wi), 0x4B400000)), 12582912.f);
                            acc[j][wi]     = __fmaf_rn(d, f0, acc[j][wi]);
                            acc[j][4 + wi] = __fmaf_rn(d, f1, acc[j][4 + wi]);
                        }
                    }
                }
            } else {
#pragma unroll
            for (int j = 0; j < PB_TOK; j++) {                 // (unrolled: acc[j] stays in registers)
                const uint8_t * r = stage + w_bytes + (size_t) (warp * PB_TOK + j) * rb;
                ActSmem A;
                A.q = (int8_t *) r; A.dx = (float *) (r + 256); A.bp = (int *) (r + 272); A.as = (int *) (r + 304);
                {
                    BlockInts bi;
                    tile_ints<TYPE>(stage, lane, 0, A, bi);
                    // chain step in registers, strictly in block order (the per-token kernel's CHAIN_REGS arithmetic)
#pragma unroll
                    for (int c = 0; c < 8; c++) acc[j][c] = __fmaf_rn(bi.d, (float) bi.s[c], acc[j][c]);
                    if (TYPE == T_Q4_K) {
#pragma unroll
                        for (int l = 0; l < 4; l++) acc[j][8 + l] = __fmaf_rn(bi.dmin, (float) bi.p[l], acc[j][8 + l]);
                    } else if (TYPE == T_Q5_K) {
                        acc[j][8] = __fadd_rn(acc[j][8], __fmul_rn(bi.dmin, (float) (bi.p[0] + bi.p[1] + bi.p[2] + bi.p[3])));
                    }
                }
            }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty0 + 8 * s);        // this warp is done with the stage
            if (tid == 0 && step + PB_STAGES < n_steps) {
                mbar_wait(empty0 + 8 * s, par);                // every warp is: refill it
                issue(step + PB_STAGES);
            }
        }
#pragma unroll
        for (int j = 0; j < PB_TOK; j++) {
            const float val = finish_row<TYPE>(acc[j]);
            pb_epilogue(a, val, ud.row0 + lane, lane, chunk * PB_CHUNK + warp * PB_TOK + j);
        }
    };
    switch (ud.type) {
        case T_Q4_K: body(TypeTag<T_Q4_K>{}); break;
        case T_Q5_K: body(TypeTag<T_Q5_K>{}); break;
        case T_Q6_K: body(TypeTag<T_Q6_K>{}); break;
        default:     body(TypeTag<T_Q8_0>{}); break;
    }
}

}  // namespace b200
