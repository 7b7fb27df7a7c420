// The router product of a batch on the tensor cores: y[t][e] = scale * sum_h x[t][h] W[e][h] with fp32 operands,
// for more than 256 tokens (512 in modes 0 and 2 of q4_cuda_mmq_tc_mode; below that the matrix-vector kernels keep a
// row's bits independent of the batch).
//
// Arithmetic: an fp32 value is the exact sum of three bf16 values, x = x1 + x2 + x3 (8 bits of mantissa each).  Of
// the nine products of the parts the six down to 2^-18 of the largest are formed (the other three are below the last
// bit of an fp32 product), each exact in the tensor core's fp32 accumulation.  Because a tensor core does not round
// its additions to nearest, the large products (x1 W1) have an accumulator of their own, an accumulator takes 128 h only,
// and both are then added to fp32 registers on the CUDA cores (one accumulator for all six: 2.2 times the largest error of 257 x 48 logits).  The logits are as close to the exact product as those of the fp32 kernel it replaces, whose 2048 terms were
// added one after the other, and there is no common scale per row, so a row with an outlier keeps its small values.
// A logit that does not come out finite is formed again as that kernel did.
//
// The fp32 kernel was bound by shared-memory bandwidth (three 16-byte loads per 32 multiply-adds): 130 us for 2048 x 512
// x 2048, 445 for 8192 tokens; this one takes 50 and 192.  A CTA here owns 128 tokens x 64 experts; its 8 warps load, split and store both
// operands of a step of 64 h (12 float4 a thread, the next step's in registers) while the MMAs of the steps before run.
#include "q4b_internal.cuh"

#include <cuda_bf16.h>

namespace rtc {

constexpr uint32_t NT = 256, BM = 128, BN = 64, KS = 64;
constexpr uint32_t A_PLANE = BM * 128u, B_PLANE = BN * 128u;            // [row][64 h], 128-byte swizzle
constexpr uint32_t BUF = 3u * (A_PLANE + B_PLANE), SMEM = 2u * BUF + 1024u;
constexpr uint32_t ERR_ROUTER = 0x2000u;

// An operand that is infinite, or that bf16 rounds to infinity, leaves NaN in the parts that remain of it, and partial
// products may overflow where their sum does not: the logits of a token's 32 experts that did not come out finite are formed
// again as fp32 sums.  (Not inlined: unrolled in the kernel it cost every call 6 us.)
__device__ __noinline__ void plain_logits(const float *W, uint32_t nrows, uint32_t ncols, const float *x, float *y, uint32_t c0,
                                          float scale) {
    for (uint32_t i = 0; i < 32u && c0 + i < nrows; i++) {
        if (isfinite(y[i])) continue;
        const float *w = W + (uint64_t)(c0 + i) * ncols;
        float v = 0.f;
        for (uint32_t h = 0; h < ncols; h++) v = fmaf(x[h], w[h], v);
        y[i] = scale * v;
    }
}

__global__ void __launch_bounds__(NT, 1) router_tc_k(const float *__restrict__ W, uint32_t nrows, uint32_t ncols,
                                                     const float *__restrict__ X, uint32_t n_tok, float *__restrict__ Y,
                                                     float scale, uint32_t *__restrict__ err) {
    using namespace mmqtc;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ unsigned long long bar[2];
    __shared__ uint32_t tmem_s;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t e0 = blockIdx.x * BN, t0 = blockIdx.y * BM, nk = 2u * ((ncols + 2u * KS - 1u) / (2u * KS));
    if (tid == 0) {
        mbar_init(&bar[0], 1), mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)), "r"(4u * BN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_s, idesc = instr_desc(BN) | (1u << 7) | (1u << 10);   // bf16 operands
    // loads: a warp takes two rows of 64 h at a time; rows past the end are zeros
    const uint32_t l_row = 2u * warp + (lane >> 4), l_c = lane & 15u;
    const uint32_t l_off = ((((l_c >> 1) ^ (l_row & 7u)) << 4) | ((l_c & 1u) << 3)) + l_row * 128u;   // + 16 rows: + 2048
    float4 ra[8], rb[4];
    auto load = [&](uint32_t ks) {
        const bool in = ks * KS + 4u * l_c < ncols;    // (past the last column: zeros, up to a whole accumulator's 128)
#pragma unroll
        for (uint32_t i = 0; i < 8; i++) {
            const uint32_t t = t0 + l_row + 16u * i;
            ra[i] = in && t < n_tok ? __ldg(reinterpret_cast<const float4 *>(X + (uint64_t)t * ncols + ks * KS) + l_c)
                              : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
            const uint32_t e = e0 + l_row + 16u * i;
            rb[i] = in && e < nrows ? __ldg(reinterpret_cast<const float4 *>(W + (uint64_t)e * ncols + ks * KS) + l_c)
                              : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto split = [&](float4 v, uint8_t *p, uint32_t plane) {
#pragma unroll
        for (uint32_t i = 0; i < 3; i++) {
            const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
            *reinterpret_cast<uint2 *>(p + i * plane) =
                make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
            const float2 fa = __bfloat1622float2(a), fb = __bfloat1622float2(b);
            v.x -= fa.x, v.y -= fa.y, v.z -= fb.x, v.w -= fb.y;   // exact
        }
    };
    bool dead = false;
    auto wait = [&](uint32_t b, uint32_t parity) {
        if (mbar_look(&bar[b], parity) || dead) return;
        unsigned long long s, t;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(s));
        do {
            if (mbar_look(&bar[b], parity)) return;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        } while (t - s < 500000000ull);
        atomicOr(err, ERR_ROUTER);
        dead = true;
    };
    float acc[32];
#pragma unroll
    for (int i = 0; i < 32; i++) acc[i] = 0.f;
    const uint32_t e_addr = tmem + ((32u * (warp & 3u)) << 16) + 32u * (warp >> 2);
    auto fold = [&](uint32_t which) {
        tc_fence_after();
        uint32_t v[32], w[32];     // the large products' sums, the small ones'
        const uint32_t at = e_addr + which * 2u * BN;
        tmem_ld16(at, v), tmem_ld16(at + 16u, v + 16);
        tmem_ld16(at + BN, w), tmem_ld16(at + BN + 16u, w + 16);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i++) acc[i] += __uint_as_float(v[i]) + __uint_as_float(w[i]);
        tc_fence_before();
    };
    load(0);
    for (uint32_t ks = 0; ks < nk; ks++) {
        const uint32_t b = ks & 1u;
        uint8_t *const buf = smem_raw + b * BUF;
        if (ks >= 2u) wait(b, ((ks >> 1) - 1u) & 1u);                 // step ks - 2 has read its operands
        if (ks >= 3u && b) fold(((ks - 2u) >> 1) & 1u);                // ... and completed 128 h
#pragma unroll
        for (uint32_t i = 0; i < 8; i++) split(ra[i], buf + l_off + 2048u * i, A_PLANE);
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) split(rb[i], buf + 3u * A_PLANE + l_off + 2048u * i, B_PLANE);
        if (ks + 1u < nk) load(ks + 1u);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (warp == 0 && elect_one()) {
            tc_fence_after();
            const uint64_t d0 = smem_desc_sw128(smem_u32(smem_raw));
            const uint32_t hi = (uint32_t)(d0 >> 32), a_lo = (uint32_t)d0 + b * (BUF >> 4), b_lo = a_lo + ((3u * A_PLANE) >> 4);
            const uint32_t d = tmem + ((ks >> 1) & 1u) * 2u * BN;
            constexpr uint32_t pa[6] = {0, 2, 1, 0, 1, 0}, pb[6] = {2, 0, 1, 1, 0, 0};   // small products first
#pragma unroll
            for (uint32_t k = 0; k < KS / 16u; k++)
#pragma unroll
                for (uint32_t p = 0; p < 6; p++)
                    mma_f16(p == 5u ? d : d + BN, desc64(a_lo + pa[p] * (A_PLANE >> 4) + 2u * k, hi), desc64(b_lo + pb[p] * (B_PLANE >> 4) + 2u * k, hi),
                            idesc, k || (p && p < 5u) ? 1u : (ks & 1u));
            mma_commit(&bar[b]);
        }
    }
    wait(1u, ((nk - 1u) >> 1) & 1u);
    fold(((nk - 1u) >> 1) & 1u);
    const uint32_t t = t0 + 32u * (warp & 3u) + lane, c0 = e0 + 32u * (warp >> 2);
    if (t < n_tok) {
        float *y = Y + (uint64_t)t * nrows + c0;
        if ((nrows & 3u) == 0 && c0 + 32u <= nrows) {
#pragma unroll
            for (int i = 0; i < 32; i += 4)
                *reinterpret_cast<float4 *>(y + i) = make_float4(scale * acc[i], scale * acc[i + 1], scale * acc[i + 2], scale * acc[i + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < 32; i++)
                if (c0 + i < nrows) y[i] = scale * acc[i];
        }
        float z = 0.f;
#pragma unroll
        for (int i = 0; i < 32; i++) z = fmaf(acc[i], 0.f, z);
        if (z != 0.f) plain_logits(W, nrows, ncols, X + (uint64_t)t * ncols, y, c0, scale);   // NaN: one is not finite
    }
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(4u * BN) : "memory");
    }
}

static bool g_ready = false;
}  // namespace rtc

bool q4b_router_tc_warm() {
    rtc::g_ready = cudaFuncSetAttribute(rtc::router_tc_k, cudaFuncAttributeMaxDynamicSharedMemorySize, rtc::SMEM) == cudaSuccess;
    if (!rtc::g_ready) cudaGetLastError();
    return rtc::g_ready;
}
// false: not this kernel's shape, nothing queued
bool q4b_router_tc(const float *W, uint64_t nrows, uint64_t ncols, const float *x, float *y, float scale, uint32_t n_tok) {
    if (!rtc::g_ready || (ncols % 4u) || ncols > 0xffffffffull || nrows > 65535ull * rtc::BN || n_tok > 65535u * rtc::BM ||
        (((uintptr_t)W | (uintptr_t)x | (uintptr_t)y) & 15u))
        return false;
    const dim3 grid((unsigned)((nrows + rtc::BN - 1) / rtc::BN), (n_tok + rtc::BM - 1) / rtc::BM);
    rtc::router_tc_k<<<grid, rtc::NT, rtc::SMEM, g_q4b.stream>>>(W, (uint32_t)nrows, (uint32_t)ncols, x, n_tok, y, scale, g_q4b.err_d);
    return true;
}
