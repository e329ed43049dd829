// attn_cluster.cuh — one token's attention of a layer in one launch: a cluster of CL blocks per KV head. BIT-EXACT with the reference's CPU arithmetic (scores as k_attn_scores,
// soft-max and P.V as k_attn_softmax_pv: tinyBLAS / ggml_vec_dot_f16 lanes, ggml_v_expf, 16 ordered chains per output).
//
// The reference's two orders ask for two cuts of the positions. A score's vector sums run over 16 consecutive ones, an output's chain c over t = c, c + 16, ...: block r scores and
// exponentiates n / CL consecutive positions (its keys are read once, nobody repeats an exponential), and walks 16 / CL chains over all of them, for all 128 dims (whole 256-byte rows of
// V). What passes between the blocks goes through distributed shared memory: the heads' maxima, the sums (double), every exponential to the block whose chain it belongs to, the chains'
// results to the block that adds them. Keys and values come through one ring of 64-row stages by asynchronous copies, values behind the keys; all but this token's own rows are asked
// for ahead of griddepcontrol.wait.
// What bounds it: four meetings of the cluster (about a microsecond each with what stands between them) and, as contexts grow, the walks themselves on the SMs that a cluster of 8 per KV
// head covers (clusters of 16 with a block per SM do not fit this GPU eight at a time): scores of 64 keys 1.4 us a block, 64 positions of P.V 1 us. A token of an 8B model's 8 layers in
// Q8_0 at 333: 515 us with two launches a layer, 489 here; at 2000 in Q4_K_M 472 and 485, at 8123 653 and 766, where the two launches stay (attn_cluster_pays).
#pragma once
#include "kernels.cuh"

namespace b200 {

static constexpr int AC_THREADS = 512, AC_ROWS = 64, AC_STRIDE = 288;                // rows of a stage; bytes between keys in it (two of a half-warp's never meet in a bank)
static constexpr int AC_STAGE = AC_ROWS * AC_STRIDE;
static constexpr int AC_STAGES[] = { 3, 4, 6, 8, 11 };                               // a ring's sizes: what the context needs, or the most that fits
static constexpr size_t AC_SMEM = 110 * 1024;
// floats beside the ring: scores of the block's own positions [GQA][own], weights of its chains [chains][GQA][n16], queries, chains' results [16][GQA][128 / CL]
__host__ __device__ constexpr int ac_own(int n16, int cl) { return (n16 + cl - 1) / cl * 16; }
__host__ __device__ constexpr int ac_row(int n16) { return (n16 + 3) / 4 * 4; }
__host__ __device__ constexpr size_t ac_beside(int gqa, int cl, int n16) { return ((size_t) gqa * ac_own(n16, cl) + (size_t) (16 / cl) * gqa * ac_row(n16) + gqa * 128 + 16 * gqa * (128 / cl)) * 4; }

__device__ __forceinline__ uint32_t ac_at(uint32_t addr, uint32_t rank) { uint32_t r; asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank)); return r; }
__device__ __forceinline__ void ac_put(uint32_t addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ void ac_put2(uint32_t addr, float u, float v) { asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" :: "r"(addr), "f"(u), "f"(v) : "memory"); }
__device__ __forceinline__ void ac_put_d(uint32_t addr, double v) { asm volatile("st.shared::cluster.f64 [%0], %1;" :: "r"(addr), "d"(v) : "memory"); }
__device__ __forceinline__ void ac_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void ac_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// all but the newest stages - 2 groups of copies have landed
__device__ __forceinline__ void ac_wait_stage(int stages) {
    switch (stages) {
        case 3: cp_async_wait<1>(); break;
        case 4: cp_async_wait<2>(); break;
        case 6: cp_async_wait<4>(); break;
        case 8: cp_async_wait<6>(); break;
        default: cp_async_wait<9>(); break;
    }
}

// grid (CL, n_head_kv), clusters of CL; n16_cap: 16-position vectors the shared memory is laid out for
// GQA: 4 or 8
template <int GQA, int CL>
__global__ void __launch_bounds__(AC_THREADS, 1) k_attn_cluster(const AttnArgs a, int n16_cap, int stages) {
    constexpr int HD = 128, CPC = 16 / CL, SLICE = HD / CL, PARTS = AC_THREADS / 32 / GQA;        // chains per block, dims it adds up, warps per head
    constexpr int HPT = 64 * CPC * GQA > AC_THREADS ? 64 * CPC * GQA / AC_THREADS : 1;      // P.V: heads of a thread
    constexpr int HG = GQA / 2;                                // scores: heads of a half of the block
    extern __shared__ __align__(128) uint8_t ac_smem[];
    __shared__ float wmax[GQA][PARTS], maxs[CL][GQA];
    __shared__ double wsum[GQA][PARTS], sums[CL][GQA];
    uint8_t * ring = ac_smem;
    float * sc = reinterpret_cast<float *>(ac_smem + (size_t) stages * AC_STAGE);    // [GQA][own]
    const int own_cap = ac_own(n16_cap, CL), prow = ac_row(n16_cap);
    float * ps = sc + GQA * own_cap;                                                  // [CPC][GQA][prow]
    float * qs = ps + CPC * GQA * prow;                                               // [GQA][HD]
    float * red = qs + GQA * HD;                                                      // [16][GQA][SLICE]
    const int r = blockIdx.x, g = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    ac_arrive();                                               // (met again before the first write into another block)
    trace_mark<true>(a.trace, 0);
    int n_kv, cur, managed = 0;                                // DecodeState is written by the previous token's last kernel
    if (a.n_kv_override > 0) { n_kv = a.n_kv_override; cur = n_kv - 1; }
    else { const int4 s1 = *(reinterpret_cast<const int4 *>(a.st) + 1); cur = s1.x; n_kv = s1.y; managed = s1.z; }
    const int n16 = (n_kv + 31) / 32 * 2, v0 = r * n16 / CL, nvec = (r + 1) * n16 / CL - v0, own = 16 * nvec, t_own = 16 * v0;
    const int nk = (own + AC_ROWS - 1) / AC_ROWS, total = nk + (n16 * CPC + AC_ROWS - 1) / AC_ROWS;
    const __half * kg = a.k_cache + g * HD, * vg = a.v_cache + g * HD;
    // stage i of the ring: 64 keys of the block's own positions, or 64 rows of V of its chains, (position / 16, chain) after one another. skip: a position that is left out
    const auto issue = [&](int i, int skip) {
        if (i < total) {
            uint8_t * slot = ring + (size_t) (i % stages) * AC_STAGE;
#pragma unroll
            for (int u = 0; u < AC_ROWS * 16 / AC_THREADS; u++) {
                const int at = tid + u * AC_THREADS, j = at >> 4, c16 = at & 15;
                if (i < nk) {
                    const int t = t_own + i * AC_ROWS + j;
                    if (i * AC_ROWS + j < own && t < n_kv && t != skip) cp_async16(slot + j * AC_STRIDE + c16 * 16, kg + (size_t) t * a.kv_dim + c16 * 8);
                } else {
                    const int row = (i - nk) * AC_ROWS + j, t = row / CPC * 16 + r * CPC + row % CPC;
                    if (t >= n_kv) *reinterpret_cast<uint4 *>(slot + j * 256 + c16 * 16) = make_uint4(0u, 0u, 0u, 0u);      // p is 0 there, and 0 x V must be
                    else if (t != skip) cp_async16(slot + j * 256 + c16 * 16, vg + (size_t) t * a.kv_dim + c16 * 8);
                }
            }
        }
        cp_async_commit();
    };
    for (int i = 0; i < stages - 1; i++) issue(i, cur);
    pdl_wait();                                                // q and this token's rows come from the QKV kernel
    pdl_launch_dependents();
    trace_mark<true>(a.trace, 1);
    if (tid < 32) {                                            // this token's rows, where their stage has been asked for
        const int c16 = tid & 15;
        if (tid < 16) {
            const int j = cur - t_own;
            if (j >= 0 && j < own && j / AC_ROWS < stages - 1)
                *reinterpret_cast<uint4 *>(ring + (size_t) (j / AC_ROWS) * AC_STAGE + (j % AC_ROWS) * AC_STRIDE + c16 * 16) = *reinterpret_cast<const uint4 *>(kg + (size_t) cur * a.kv_dim + c16 * 8);
        } else {
            const int c = cur % 16 - r * CPC, row = cur / 16 * CPC + c, i = nk + row / AC_ROWS;
            if (c >= 0 && c < CPC && i < stages - 1)
                *reinterpret_cast<uint4 *>(ring + (size_t) i * AC_STAGE + (row % AC_ROWS) * 256 + c16 * 16) = *reinterpret_cast<const uint4 *>(vg + (size_t) cur * a.kv_dim + c16 * 8);
        }
    }
    int round_q = a.round_q_override, pos = 0;
    if (a.st) { const int4 s0 = *reinterpret_cast<const int4 *>(a.st); pos = s0.y; round_q = s0.z; }
    for (int i = tid; i < GQA * HD; i += AC_THREADS) {
        float v = a.q[(size_t) (g * GQA) * HD + i];
        if (round_q) v = __half2float(__float2half_rn(v));    // src1 converted to the vec_dot_type F16 (ggml.c:12345-12371)
        qs[i] = v;
    }
    // ---- scores: four lanes a key (k_attn_scores has the arithmetic)
    const int key = (tid & 255) >> 2, c4 = tid & 3, hg = tid >> 8;
    for (int i = 0; i < nk; i++) {
        ac_wait_stage(stages);
        __syncthreads();
        issue(i + stages - 1, -1);
        const int at = i * AC_ROWS + key, t = t_own + at;
        bool visible = at < own && t < n_kv;
        if (managed && visible) { const int p = a.cell_pos[t]; visible = p >= 0 && p <= pos; }
        const uint8_t * kr = ring + (size_t) (i % stages) * AC_STAGE + key * AC_STRIDE + 8 * c4;
        float kf[8][4];
#pragma unroll
        for (int s = 0; s < 8; s++) {
            const uint2 kv = *reinterpret_cast<const uint2 *>(kr + 32 * s);
            const float2 f0 = __half22float2(*reinterpret_cast<const __half2 *>(&kv.x)), f1 = __half22float2(*reinterpret_cast<const __half2 *>(&kv.y));
            kf[s][0] = f0.x; kf[s][1] = f0.y; kf[s][2] = f1.x; kf[s][3] = f1.y;
        }
        {
#pragma unroll 1
            for (int h = hg * HG; h < (hg + 1) * HG; h++) {
                const float * q = qs + h * HD;
                float ch[4];
                if (!round_q) {
                    // tinyBLAS<16>: lane c: acc = fma(k[16s+c], q[16s+c], acc), s = 0..7
#pragma unroll
                    for (int e = 0; e < 4; e++) ch[e] = 0.f;
#pragma unroll
                    for (int s = 0; s < 8; s++) {
                        const float4 qv = *reinterpret_cast<const float4 *>(q + 16 * s + 4 * c4);
                        ch[0] = __fmaf_rn(kf[s][0], qv.x, ch[0]); ch[1] = __fmaf_rn(kf[s][1], qv.y, ch[1]);
                        ch[2] = __fmaf_rn(kf[s][2], qv.z, ch[2]); ch[3] = __fmaf_rn(kf[s][3], qv.w, ch[3]);
                    }
                } else {
                    // ggml_vec_dot_f16: sum[j][c] over i in {0, 64}: element i + 16j + c; then (0+2)+(1+3)
                    float aj[4][4];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float4 q0 = *reinterpret_cast<const float4 *>(q + 16 * j + 4 * c4), q1 = *reinterpret_cast<const float4 *>(q + 64 + 16 * j + 4 * c4);
                        aj[j][0] = __fmaf_rn(kf[4 + j][0], q1.x, __fmul_rn(kf[j][0], q0.x));
                        aj[j][1] = __fmaf_rn(kf[4 + j][1], q1.y, __fmul_rn(kf[j][1], q0.y));
                        aj[j][2] = __fmaf_rn(kf[4 + j][2], q1.z, __fmul_rn(kf[j][2], q0.z));
                        aj[j][3] = __fmaf_rn(kf[4 + j][3], q1.w, __fmul_rn(kf[j][3], q0.w));
                    }
#pragma unroll
                    for (int e = 0; e < 4; e++) ch[e] = __fadd_rn(__fadd_rn(aj[0][e], aj[2][e]), __fadd_rn(aj[1][e], aj[3][e]));
                }
                // _mm512_reduce_add_ps over the 16 chains: lanes c4 = 0..3 hold chains 4 c4 .. 4 c4 + 3
                float t3[4], t6[4];
#pragma unroll
                for (int e = 0; e < 4; e++) t3[e] = __fadd_rn(__shfl_xor_sync(0xffffffffu, ch[e], 2), ch[e]);
#pragma unroll
                for (int e = 0; e < 4; e++) t6[e] = __fadd_rn(__shfl_xor_sync(0xffffffffu, t3[e], 1), t3[e]);
                const float res = __fadd_rn(__fadd_rn(t6[0], t6[2]), __fadd_rn(t6[1], t6[3]));
                if (c4 == 0 && at < own) sc[h * own_cap + at] = visible ? __fmul_rn(res, a.scale) : -INFINITY;
            }
        }
    }
    __syncthreads();
    trace_mark<true>(a.trace, 2);
    // ---- the heads' maxima, over all blocks
    const int h = warp % GQA, part = warp / GQA;
    const float * row = sc + h * own_cap;
    {
        float mx = -INFINITY;
        for (int i = part * 32 + lane; i < own; i += 32 * PARTS) mx = fmaxf(mx, row[i]);
        mx = warp_max(mx);
        if (lane == 0) wmax[h][part] = mx;
        __syncthreads();
        ac_wait();                                             // every block of the cluster runs
        if (tid < GQA * CL) {
            const int hh = tid % GQA;
            float m = wmax[hh][0];
#pragma unroll
            for (int i = 1; i < PARTS; i++) m = fmaxf(m, wmax[hh][i]);
            ac_put(ac_at(smem_u32(&maxs[r][hh]), (uint32_t) (tid / GQA)), m);
        }
    }
    __syncwarp();
    ac_arrive();
    ac_wait();
    // ---- exponentials of the block's own vectors, each to the block whose chain it belongs to; their sums (soft_max_ext, cpp/ggml/src/ggml.c:13682-13778; see k_attn_softmax)
    float mx = maxs[0][h];
#pragma unroll
    for (int i = 1; i < CL; i++) mx = fmaxf(mx, maxs[i][h]);
    double part_sum = 0.0;
    {
        const int rot = (lane >> 1) & 3;                       // k_attn_softmax_pv: the lanes of a quarter-warp start in different banks, no bit of the sum changes
        const uint32_t base = smem_u32(ps + h * prow);
        for (int v = part * 32 + lane; v < nvec; v += 32 * PARTS) {
            const float4 * r4 = reinterpret_cast<const float4 *>(row + 16 * v);
            float4 t[2];
#pragma unroll 1
            for (int pq = 0; pq < 2; pq++) {
                const int f0 = (pq + rot) & 3, f1 = f0 ^ 2;
                float4 lo = r4[f0], hi = r4[f1];
                lo.x = v_expf(__fsub_rn(lo.x, mx)); lo.y = v_expf(__fsub_rn(lo.y, mx)); lo.z = v_expf(__fsub_rn(lo.z, mx)); lo.w = v_expf(__fsub_rn(lo.w, mx));
                hi.x = v_expf(__fsub_rn(hi.x, mx)); hi.y = v_expf(__fsub_rn(hi.y, mx)); hi.z = v_expf(__fsub_rn(hi.z, mx)); hi.w = v_expf(__fsub_rn(hi.w, mx));
                const float e[8] = { lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w };
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const int c = 4 * (k < 4 ? f0 : f1) + (k & 3);
                    ac_put(ac_at(base + (uint32_t) ((c % CPC) * GQA * prow + v0 + v) * 4u, (uint32_t) (c / CPC)), e[k]);
                }
                const float4 tt = make_float4(__fadd_rn(hi.x, lo.x), __fadd_rn(hi.y, lo.y), __fadd_rn(hi.z, lo.z), __fadd_rn(hi.w, lo.w));
                if (f0 & 1) t[1] = tt; else t[0] = tt;
            }
            const float u0 = __fadd_rn(t[1].x, t[0].x), u1 = __fadd_rn(t[1].y, t[0].y), u2 = __fadd_rn(t[1].z, t[0].z), u3 = __fadd_rn(t[1].w, t[0].w);
            part_sum += (double) __fadd_rn(__fadd_rn(u0, u2), __fadd_rn(u1, u3));
        }
    }
    part_sum = warp_sum_d(part_sum);
    if (lane == 0) wsum[h][part] = part_sum;
    __syncthreads();
    if (tid < GQA * CL) {
        const int hh = tid % GQA;
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < PARTS; i++) s += wsum[hh][i];
        ac_put_d(ac_at(smem_u32(&sums[r][hh]), (uint32_t) (tid / GQA)), s);
    }
    __syncwarp();
    ac_arrive();
    ac_wait();
    trace_mark<true>(a.trace, 3);
    {   // this block's weights: e x (1 / sum)
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < CL; i++) s += sums[i][h];
        const float inv = (float) (1.0 / s);
#pragma unroll
        for (int cc = 0; cc < CPC; cc++)
            for (int v = part * 32 + lane; v < n16; v += 32 * PARTS) { float & p = ps[(cc * GQA + h) * prow + v]; p = __fmul_rn(p, inv); }
    }
    // ---- P.V: acc = fma(V[t][d], p[t], acc) over t = c, c + 16, ...: a thread has one chain, two dims, HPT heads
    const int dp = tid % 64, cc = tid / 64 % CPC, h0 = tid / (64 * CPC) * HPT;
    float acc[HPT][2] = {};
    for (int i = nk; i < total; i++) {
        ac_wait_stage(stages);
        __syncthreads();
        issue(i + stages - 1, -1);
        if (h0 < GQA) {
            const int vb = (i - nk) * (AC_ROWS / CPC), cnt = min(AC_ROWS / CPC, n16 - vb);
            const uint8_t * vr = ring + (size_t) (i % stages) * AC_STAGE + cc * 256 + dp * 4;
            const float * pr = ps + (size_t) (cc * GQA + h0) * prow + vb;
            int j = 0;
#pragma unroll 2
            for (; j + 4 <= cnt; j += 4) {
                float4 p4[HPT];
                float2 v[4];
#pragma unroll
                for (int k = 0; k < HPT; k++) p4[k] = *reinterpret_cast<const float4 *>(pr + k * prow + j);
#pragma unroll
                for (int u = 0; u < 4; u++) v[u] = __half22float2(*reinterpret_cast<const __half2 *>(vr + (j + u) * (CPC * 256)));
#pragma unroll
                for (int u = 0; u < 4; u++) {
#pragma unroll
                    for (int k = 0; k < HPT; k++) {
                        const float p = u == 0 ? p4[k].x : u == 1 ? p4[k].y : u == 2 ? p4[k].z : p4[k].w;
                        acc[k][0] = __fmaf_rn(v[u].x, p, acc[k][0]); acc[k][1] = __fmaf_rn(v[u].y, p, acc[k][1]);
                    }
                }
            }
            for (; j < cnt; j++) {
                const float2 v = __half22float2(*reinterpret_cast<const __half2 *>(vr + j * (CPC * 256)));
#pragma unroll
                for (int k = 0; k < HPT; k++) { const float p = pr[k * prow + j]; acc[k][0] = __fmaf_rn(v.x, p, acc[k][0]); acc[k][1] = __fmaf_rn(v.y, p, acc[k][1]); }
            }
        }
    }
    if (h0 < GQA) {
#pragma unroll
        for (int k = 0; k < HPT; k++)
            ac_put2(ac_at(smem_u32(red + ((r * CPC + cc) * GQA + h0 + k) * SLICE + 2 * dp % SLICE), (uint32_t) (2 * dp / SLICE)), acc[k][0], acc[k][1]);
    }
    __syncwarp();
    ac_arrive();
    ac_wait();
    trace_mark<true>(a.trace, 4);
    if (tid < GQA * SLICE) {
        const int hh = tid / SLICE, dd = tid % SLICE;
        const float * x = red + hh * SLICE + dd;
        float t3[8], t6[4];                                   // _mm512_reduce_add_ps over the 16 chains
#pragma unroll
        for (int j = 0; j < 8; j++) t3[j] = __fadd_rn(x[(8 + j) * GQA * SLICE], x[j * GQA * SLICE]);
#pragma unroll
        for (int j = 0; j < 4; j++) t6[j] = __fadd_rn(t3[4 + j], t3[j]);
        a.out[(size_t) (g * GQA + hh) * HD + r * SLICE + dd] = __fadd_rn(__fadd_rn(t6[0], t6[2]), __fadd_rn(t6[1], t6[3]));     // kqv_merged_cont layout: [n_head*hd]
    }
}

}  // namespace b200
