// stack_kernels_f32.cuh — float32 products on the tensor cores (sm_100a, tcgen05): Y = X W^T (+ bias), the operand layouts of k_gemm_simt_big.
//
// The method is that of Henry, Tang and Heinecke (Leveraging the bfloat16 artificial intelligence datatype for higher-precision computations, 2019).
// A float32 number is the sum of three bfloat16 ones, exactly: hi = bf16(x), mid = bf16(x - hi), lo = x - hi - mid (24 bits are 8 + 8 + 8; a number below 2^-110 loses what is below 2^-133).
// A product of two takes six MMAs (hi hi, hi mid, mid hi, mid mid, hi lo, lo hi; what is left out is below 2^-26 of it). The tensor cores add in float32 without rounding to
// nearest, so an accumulator holds 64 terms of a sum only: the small products first, hi hi last, then it is added to registers. Against 64 bits that is as close as a
// chain of fmaf or closer (2-norm, random operands of nine shapes, k 64 to 8192: 0.8e-7 to 1.6e-7 here, 1.2e-7 to 5.7e-7 by fmaf; a whole float32 model's logits 4.5e-7 and 1.1e-6).
//   workers   16 warps: float32 slices of both operands from global memory (the next one's loads in flight), split, 16-bit planes into shared memory in the 128-byte swizzle;
//             then the sums of the slice before last out of tensor memory (two accumulators) into registers
//   MMA warp  24 tcgen05.mma of 128 x 128 x 16 per slice of 64 k
// What bounds it: one block per SM whose slice is a chain (load, split and store, hand-over, MMAs, drain) that two stages overlap in part only: under ncu 50 % of the issue slots and
// 23 to 31 % of the tensor pipe are busy (512 x 8192 x 1024 in 84 us). The MMAs alone, 65 clocks each, would allow 375 TFLOP/s of float32 products; 600 x 16000 x 1024 reach 126.
// Measured (B200), the fp32 pipe's tiles and this: 600 x 16000 x 1024 694 and 156 us, 300 x 4096 x 1024 91 and 35, 64 x 512 x 512 40 and 16; scores of 512 tokens x 16 heads over
// windows of 1152 rows of 576 260 and 92.
// Rows and columns of a tile with an infinity or a NaN (whose parts would be NaN) are done again by fmaf, and they alone: what an output is does not depend on the rows beside it.
// The loop only notices that there is one; a tile that has one looks for its rows then (largest magnitudes kept per row in the loop: 4 us a tile more). What a number below
// 2^-110 loses, less than 2^-133, is left: attention weights of far keys are such numbers, and beside their row's others it is nothing.
#pragma once

namespace b200 {
namespace stk {

constexpr int F3_BM = 128, F3_BN = 128, F3_BK = 64, F3_WORKERS = 512, F3_THREADS = F3_WORKERS + 32;
constexpr int F3_PLANE = 128 * F3_BK * 2, F3_STAGE = 6 * F3_PLANE, F3_SMEM = 2 * F3_STAGE + 1024;       // X hi, mid, lo | W hi, mid, lo; + alignment slack

// two numbers into a word of each plane; odd turns NaN with a number that is not finite as bfloat16
__device__ __forceinline__ void f3_split(float x, float y, uint32_t & hi, uint32_t & mid, uint32_t & lo, float & odd) {
    hi = pack_bf16(x, y);
    const float rx = x - __uint_as_float(hi << 16), ry = y - __uint_as_float(hi & 0xffff0000u);
    mid = pack_bf16(rx, ry);
    const float lx = rx - __uint_as_float(mid << 16), ly = ry - __uint_as_float(mid & 0xffff0000u);
    lo = __byte_perm(__float_as_uint(lx), __float_as_uint(ly), 0x7632u);
    odd = fmaf(lx, 0.f, fmaf(ly, 0.f, odd));
}

// What a warp of a tile with odd numbers does for its 32 rows from mw and 32 columns from nb: rows and columns with a number that is not
// finite as bfloat16 are formed by fmaf, a lane per output, into again [row][33]. Returns their masks.
__device__ __noinline__ uint2 f3_again(const float * X, int ldx, const float * W, int ldw, bool w_kn, int T, int N, int kbeg, int K, int mw, int nb, float * again) {
    const int lane = threadIdx.x & 31;
    const auto off = [](uint32_t top) { return top >= 0x7f7f8000u; };                  // (from there on rounding gives infinity)
    const auto bits = [](float v) { return __float_as_uint(v) & 0x7fffffffu; };        // magnitudes and NaN are ordered as their bits
    uint32_t x_off = 0, w_off = 0;
#pragma unroll 1
    for (int i = 0; i < 32; i++) {
        uint32_t x = 0, w = 0;
        for (int k = kbeg + lane; k < K; k += 32) {
            if (mw + i < T) x = max(x, bits(X[(size_t) (mw + i) * ldx + k]));
            if (nb + i < N && !w_kn) w = max(w, bits(W[(size_t) (nb + i) * ldw + k]));
        }
        if (off(__reduce_max_sync(0xffffffffu, x))) x_off |= 1u << i;
        if (off(__reduce_max_sync(0xffffffffu, w))) w_off |= 1u << i;
    }
    if (w_kn) {
        uint32_t w = 0;
        if (nb + lane < N) for (int k = kbeg; k < K; k++) w = max(w, bits(W[(size_t) k * ldw + nb + lane]));
        w_off = __ballot_sync(0xffffffffu, off(w));
    }
    const auto chain = [&](int m, int n) {
        float v = 0.f;
        if (m >= T || n >= N) return v;
        const float * x = X + (size_t) m * ldx;
#pragma unroll 4
        for (int k = kbeg; k < K; k += 4) {             // (K is a multiple of 4)
            const float4 u = *reinterpret_cast<const float4 *>(x + k);
            float4 w;
            if (w_kn) { const float * p = W + (size_t) k * ldw + n; w = make_float4(p[0], p[ldw], p[2 * (size_t) ldw], p[3 * (size_t) ldw]); }
            else w = *reinterpret_cast<const float4 *>(W + (size_t) n * ldw + k);
            v = fmaf(u.w, w.w, fmaf(u.z, w.z, fmaf(u.y, w.y, fmaf(u.x, w.x, v))));
        }
        return v;
    };
#pragma unroll 1
    for (int i = 0; i < 32; i++) {                      // a row: lane = column, a column: lane = row
        if (x_off >> i & 1) again[i * 33 + lane] = chain(mw + i, nb + lane);
        if (w_off >> i & 1) again[lane * 33 + i] = chain(mw + lane, nb + i);
    }
    __syncwarp();
    return make_uint2(x_off, w_off);
}

__global__ void __launch_bounds__(F3_THREADS, 1) k_gemm_f32_umma(const LinArgs a, int * err, int ksplit = 1, float * part = nullptr) {
    pdl_enter();
    extern __shared__ uint8_t f3_raw[];
    __shared__ __align__(8) uint64_t full[2], done[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ int failed_s, odd_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t smem0 = (smem_addr(f3_raw) + 1023u) & ~1023u;
    uint8_t * const sm = f3_raw + (smem0 - smem_addr(f3_raw));
    const int m0 = blockIdx.y * F3_BM, n0 = blockIdx.x * F3_BN;
    const int zb = ksplit > 1 ? 0 : blockIdx.z, z1 = zb / a.nz2, z2 = zb - z1 * a.nz2;
    const int r0 = a.seg ? a.seg[zb] : 0, T = a.seg ? a.seg[zb + 1] - r0 : a.rows_all > 0 ? min(a.T, a.rows_all - z1 * a.T) : a.T;
    if (m0 >= T) return;                      // (the whole block, before anything is allocated)
    const float * X = a.X + (a.seg ? (size_t) r0 * a.ldx : (size_t) z1 * a.sX + (size_t) z2 * a.sX2);
    const float * W = reinterpret_cast<const float *>(a.W) + (size_t) z1 * a.sW + (size_t) z2 * a.sW2;
    const int ldw = a.ldw > 0 ? a.ldw : a.K;
    int K = a.K;
    if (a.see_rows > 0) {
        const int last = tile_sees(a, z1, m0, F3_BM);
        if (a.w_kn) K = min(K, (last + 4) / 4 * 4);
        else if (n0 > last) return;
    }
    int kbeg = 0;
    if (ksplit > 1) {
        const int slices = (K + F3_BK - 1) / F3_BK;
        kbeg = (int) ((long long) slices * blockIdx.z / ksplit) * F3_BK;
        K = min(K, (int) ((long long) slices * (blockIdx.z + 1) / ksplit) * F3_BK);
    }
    const int nk = (K - kbeg + F3_BK - 1) / F3_BK;      // at least one: ksplit <= slices
    volatile int * failed = &failed_s;
    if (tid == 0) {
        failed_s = 0; odd_s = 0;
        for (int s = 0; s < 2; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_addr(&full[s])), "r"(F3_WORKERS / 32) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_addr(&done[s])) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_addr(&tmem_base_s)), "r"(256u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_s;
    if (warp == F3_WORKERS / 32) {
        // instruction descriptor: D f32, A and B bf16, both K-major, N = 128, M = 128; operands K-major in the 128-byte swizzle (as in k_gemm_bf16_umma)
        constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t) (F3_BN >> 3) << 17) | ((uint32_t) (F3_BM >> 4) << 24);
        constexpr uint64_t DESC = ((uint64_t) 1 << 16) | ((uint64_t) (1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
        bool dead = false;
        for (int c = 0; c < nk; c++) {
            const int s = c & 1;
            tc_wait(smem_addr(&full[s]), (uint32_t) ((c >> 1) & 1), dead);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one() && !dead) {
                const uint32_t sx = smem0 + (uint32_t) s * F3_STAGE, sw = sx + 3 * F3_PLANE;
#pragma unroll
                for (int q = 0; q < 6; q++) {
                    constexpr int px[6] = {2, 0, 1, 1, 0, 0}, pw[6] = {0, 2, 1, 0, 1, 0};       // small products first
#pragma unroll
                    for (int ks = 0; ks < F3_BK / 16; ks++) {
                        const uint64_t da = DESC | (uint64_t) (((sx + px[q] * F3_PLANE + ks * 32u) >> 4) & 0x3fffu), db = DESC | (uint64_t) (((sw + pw[q] * F3_PLANE + ks * 32u) >> 4) & 0x3fffu);
                        const uint32_t accumulate = (q | ks) ? 1u : 0u;
                        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                                     :: "r"(tmem + (uint32_t) s * F3_BN), "l"(da), "l"(db), "r"(IDESC), "r"(accumulate) : "memory");
                    }
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_addr(&done[s])) : "memory");
            }
            __syncwarp();
        }
        if (dead) { *failed = 1; atomicExch(err, 1); for (int i = 0; i < 1000; i++) __nanosleep(1000); }      // MMAs under way end before tensor memory is given back
        __syncwarp();
    } else {
        // ---- slices. Rows of X (and of W [N][K]): 16 threads a row, four rows a thread, 4 k each; a W [K][N]: a thread a column, 16 k
        float4 xr[4];
        float wr[16];
        float odd = 0.f;
        const int lr = tid >> 4, lk = tid & 15, wn = tid & 127, wk = (tid >> 7) * 16;
        const auto fetch = [&](int k0) {
            const int k = k0 + 4 * lk;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int m = m0 + lr + 32 * i, n = n0 + lr + 32 * i;
                xr[i] = m < T && k < K ? *reinterpret_cast<const float4 *>(X + (size_t) m * a.ldx + k) : make_float4(0.f, 0.f, 0.f, 0.f);       // K is a multiple of 4
                if (!a.w_kn) {
                    const float4 v = n < a.N && k < K ? *reinterpret_cast<const float4 *>(W + (size_t) n * ldw + k) : make_float4(0.f, 0.f, 0.f, 0.f);
                    wr[4 * i] = v.x; wr[4 * i + 1] = v.y; wr[4 * i + 2] = v.z; wr[4 * i + 3] = v.w;
                }
            }
            if (a.w_kn) {
#pragma unroll
                for (int i = 0; i < 16; i++) wr[i] = n0 + wn < a.N && k0 + wk + i < K ? W[(size_t) (k0 + wk + i) * ldw + n0 + wn] : 0.f;
            }
        };
        const auto store4 = [&](uint8_t * plane0, int row, float x, float y, float z, float w) {
            uint32_t h[2], m[2], l[2];
            f3_split(x, y, h[0], m[0], l[0], odd);
            f3_split(z, w, h[1], m[1], l[1], odd);
            uint8_t * p = plane0 + row * 128 + (((lk >> 1) ^ (row & 7)) << 4) + (lk & 1) * 8;
            *reinterpret_cast<uint2 *>(p) = make_uint2(h[0], h[1]);
            *reinterpret_cast<uint2 *>(p + F3_PLANE) = make_uint2(m[0], m[1]);
            *reinterpret_cast<uint2 *>(p + 2 * F3_PLANE) = make_uint2(l[0], l[1]);
        };
        float acc[32];
#pragma unroll
        for (int j = 0; j < 32; j++) acc[j] = 0.f;
        const uint32_t taddr = tmem + ((uint32_t) (32 * (warp & 3)) << 16) + (uint32_t) (warp >> 2) * 32;      // this warp's 32 rows and 32 columns
        const auto drain = [&](int c) {
            mbar_wait_limited(smem_addr(&done[c & 1]), (uint32_t) ((c >> 1) & 1), failed, err);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int h = 0; h < 2; h++) {
                uint32_t v[16];
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                             : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]),
                               "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(taddr + (uint32_t) (c & 1) * F3_BN + 16 * h) : "memory");
                tc_ld_ready(v);
#pragma unroll
                for (int j = 0; j < 16; j++) acc[16 * h + j] += __uint_as_float(v[j]);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        };
        fetch(kbeg);
#pragma unroll 1
        for (int c = 0; c < nk; c++) {
            uint8_t * st = sm + (c & 1) * F3_STAGE;             // free: slice c - 2 was drained
#pragma unroll
            for (int i = 0; i < 4; i++) {
                store4(st, lr + 32 * i, xr[i].x, xr[i].y, xr[i].z, xr[i].w);
                if (!a.w_kn) store4(st + 3 * F3_PLANE, lr + 32 * i, wr[4 * i], wr[4 * i + 1], wr[4 * i + 2], wr[4 * i + 3]);
            }
            if (a.w_kn) {
#pragma unroll
                for (int g = 0; g < 2; g++) {
                    uint32_t h[4], m[4], l[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) f3_split(wr[8 * g + 2 * i], wr[8 * g + 2 * i + 1], h[i], m[i], l[i], odd);
                    uint8_t * p = st + 3 * F3_PLANE + wn * 128 + ((((wk >> 3) + g) ^ (wn & 7)) << 4);
                    *reinterpret_cast<uint4 *>(p) = make_uint4(h[0], h[1], h[2], h[3]);
                    *reinterpret_cast<uint4 *>(p + F3_PLANE) = make_uint4(m[0], m[1], m[2], m[3]);
                    *reinterpret_cast<uint4 *>(p + 2 * F3_PLANE) = make_uint4(l[0], l[1], l[2], l[3]);
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_addr(&full[c & 1])) : "memory");
            if (c + 1 < nk) fetch(kbeg + (c + 1) * F3_BK);
            if (c > 0) drain(c - 1);
        }
        drain(nk - 1);
        if (odd != 0.f) odd_s = 1;                              // (NaN compares unequal)
        asm volatile("bar.sync 1, %0;" :: "n"(F3_WORKERS) : "memory");
        const int mw = m0 + 32 * (warp & 3), m = mw + lane, nb = n0 + (warp >> 2) * 32;
        if (odd_s) {                                            // through the slices' memory, which the MMAs are done with
            float * again = reinterpret_cast<float *>(sm) + warp * (32 * 33);
            const uint2 off = f3_again(X, a.ldx, W, ldw, a.w_kn != 0, T, a.N, kbeg, K, mw, nb, again);
#pragma unroll
            for (int j = 0; j < 32; j++) if ((off.x >> lane | off.y >> j) & 1) acc[j] = again[lane * 33 + j];
        }
        if (m < T && !*failed) {
            const int ldy = ksplit > 1 ? a.N : a.ldy;
            const float * bias = ksplit > 1 ? nullptr : a.bias;
            float * Y = (ksplit > 1 ? part + (size_t) blockIdx.z * T * a.N : a.seg ? a.Y + (size_t) r0 * ldy : a.Y + (size_t) z1 * a.sY + (size_t) z2 * a.sY2) + (size_t) m * ldy;
            if (a.glu) {
#pragma unroll
                for (int j = 0; j < 32; j += 2)
                    if (nb + j + 1 < a.N) Y[(nb + j) >> 1] = gated_unit(a, acc[j] + (bias ? bias[nb + j] : 0.f), acc[j + 1] + (bias ? bias[nb + j + 1] : 0.f));
            } else {
                const bool wide = (ldy & 3) == 0 && ((uintptr_t) (Y + nb) & 15) == 0;
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
#pragma unroll
                    for (int i = 0; i < 4; i++) if (nb + j + i < a.N) acc[j + i] += (bias ? bias[nb + j + i] : 0.f) + (a.accum ? Y[nb + j + i] : 0.f);
                    if (wide && nb + j + 3 < a.N) *reinterpret_cast<float4 *>(Y + nb + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
                    else {
#pragma unroll
                        for (int i = 0; i < 4; i++) if (nb + j + i < a.N) Y[nb + j + i] = acc[j + i];
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(256u) : "memory");
    }
}

}  // namespace stk
}  // namespace b200
