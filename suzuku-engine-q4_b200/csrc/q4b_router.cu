// The router product of a batch on the tensor cores: y[t][e] = scale * sum_h x[t][h] W[e][h] with fp32 operands,
// for more than 256 tokens (512 in modes 0 and 2 of q4_cuda_mmq_tc_mode; below that the matrix-vector kernels keep a
// row's bits independent of the batch).
//
// Arithmetic: an fp32 value is the exact sum of three bf16 values, x = x1 + x2 + x3 (8 bits of mantissa each).  Of
// the nine products of the parts the six down to 2^-18 of the largest are formed (the other three are below the last
// bit of an fp32 product), each exact in the tensor core's fp32 accumulation.  Because a tensor core does not round
// its additions to nearest, the products of a size have an accumulator of their own (x1 W1 | x1 W2 + x2 W1 | x1 W3 + x2 W2 +
// x3 W1), an accumulator takes 128 h only, and all three are then added to fp32 registers on the CUDA cores (one accumulator
// for all six: 2.2 times the largest error of 257 x 48 logits).  The logits are as close to the exact product as those of the
// fp32 kernel it replaces, whose 2048 terms were
// added one after the other, and there is no common scale per row, so a row with an outlier keeps its small values.
// A logit that does not come out finite is formed again as that kernel did.
//
// A CTA owns 128 tokens x 64 experts; 16 warps load, split and store both operands of a step of 64 h (6 float4 a thread, the
// next step's in registers) into one of three buffers, one warp issues the MMAs.  The three parts of W lie behind one
// another, so x1 meets all of them in one MMA of N = 192, x2 two and x3 one: 24 KB of shared memory read a 16 h, with six
// MMAs 36.  Measured, 512 experts x 2048: 2048 tokens 47.9 -> 41.0 us, 8192 tokens 179 -> 160 (8 warps that also issued, six
// MMAs; the fp32 kernel before that took 130 and 445); 300 tokens x 48 experts x 1024 26.6 -> 20.9.  What bounds it: the
// splitting, 62 % of the issue slots while a tenth of the MMAs, no proxy fence or no folding change the time by 5 %, and a second
// step of loads ahead by nothing.
#include "q4b_internal.cuh"

#include <cuda_bf16.h>

namespace rtc {

constexpr uint32_t NW = 16, NT = 32 * (NW + 4), BM = 128, BN = 64, KS = 64, NBUF = 3;   // NW warps split, one issues
constexpr uint32_t A_PLANE = BM * 128u, B_PLANE = BN * 128u;            // [row][64 h], 128-byte swizzle
constexpr uint32_t BUF = 3u * (A_PLANE + B_PLANE), SMEM = NBUF * BUF + 1024u;
constexpr uint32_t ERR_ROUTER = 0x2000u;

// An operand that is infinite, or that bf16 rounds to infinity, leaves NaN in the parts that remain of it, and partial
// products may overflow where their sum does not: the logits of a token's 16 experts that did not come out finite are formed
// again as fp32 sums.  (Not inlined: unrolled in the kernel it cost every call 6 us.)
__device__ __noinline__ void plain_logits(const float *W, uint32_t nrows, uint32_t ncols, const float *x, float *y, uint32_t c0,
                                          float scale) {
    for (uint32_t i = 0; i < 16u && c0 + i < nrows; i++) {
        if (isfinite(y[i])) continue;
        const float *w = W + (uint64_t)(c0 + i) * ncols;
        float v = 0.f;
        for (uint32_t h = 0; h < ncols; h++) v = fmaf(x[h], w[h], v);
        y[i] = scale * v;
    }
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}
__global__ void __launch_bounds__(NT, 1) router_tc_k(const float *__restrict__ W, uint32_t nrows, uint32_t ncols,
                                                     const float *__restrict__ X, uint32_t n_tok, float *__restrict__ Y,
                                                     float scale, uint32_t *__restrict__ err) {
    using namespace mmqtc;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ unsigned long long full[NBUF], empty[NBUF], acc_empty[2];
    __shared__ uint32_t tmem_s;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t e0 = blockIdx.x * BN, t0 = blockIdx.y * BM, nk = 2u * ((ncols + 2u * KS - 1u) / (2u * KS));
    if (tid == 0) {
        for (uint32_t i = 0; i < NBUF; i++) mbar_init(&full[i], NW), mbar_init(&empty[i], 1);
        mbar_init(&acc_empty[0], NW), mbar_init(&acc_empty[1], NW);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)), "r"(8u * BN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_s;
    bool dead = false;
    auto wait = [&](unsigned long long *bar, uint32_t parity) {
        if (mbar_look(bar, parity) || dead) return;
        unsigned long long s, t;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(s));
        do {
            if (mbar_look(bar, parity)) return;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        } while (t - s < 500000000ull);
        atomicOr(err, ERR_ROUTER);
        dead = true;
    };
    // 96 registers a thread at launch (61,440 a CTA), shared out anew: 112 and 24 make 60,416
    if (warp >= NW) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
        // ---- the MMA warp (one lane) ----
        if (warp == NW && elect_one()) {
            const uint64_t d0 = smem_desc_sw128(smem_u32(smem_raw));
            const uint32_t hi = (uint32_t)(d0 >> 32);
            constexpr uint32_t BF16 = (1u << 7) | (1u << 10);
            uint32_t b = 0, ph = 0;
            for (uint32_t ks = 0; ks < nk; ks++) {
                const uint32_t i = ks >> 1, d = tmem + (i & 1u) * 4u * BN;       // accumulators of 128 h, by size of the products
                if (i >= 2u && (ks & 1u) == 0) wait(&acc_empty[i & 1u], ((i >> 1) - 1u) & 1u);
                wait(&full[b], ph);
                tc_fence_after();
                const uint32_t a_lo = (uint32_t)d0 + b * (BUF >> 4), b_lo = a_lo + ((3u * A_PLANE) >> 4);
#pragma unroll
                for (uint32_t k = 0; k < KS / 16u; k++)
#pragma unroll
                    for (uint32_t p = 0; p < 3; p++)      // part p of x, parts 0 .. 2 - p of W
                        mma_f16(d + p * BN, desc64(a_lo + p * (A_PLANE >> 4) + 2u * k, hi), desc64(b_lo + 2u * k, hi),
                                instr_desc((3u - p) * BN) | BF16, k || p ? 1u : (ks & 1u));
                mma_commit(&empty[b]);
                if (++b == NBUF) b = 0, ph ^= 1u;
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
        // Loads: a warp takes two rows of 64 h at a time.  Rows past the end are the last one again (their logits are not
        // stored); columns past the end, up to a whole accumulator's 128, are zeros.
        const uint32_t l_row = 2u * warp + (lane >> 4), l_c = lane & 15u;
        const uint32_t l_off = ((((l_c >> 1) ^ (l_row & 7u)) << 4) | ((l_c & 1u) << 3)) + l_row * 128u;   // + 32 rows: + 4096
        float4 va[6];                                  // the next step's: four rows of x, two of W
        const float4 *src[6];
#pragma unroll
        for (uint32_t i = 0; i < 6; i++)
            src[i] = reinterpret_cast<const float4 *>(i < 4 ? X + (uint64_t)min(t0 + l_row + 32u * i, n_tok - 1u) * ncols
                                                            : W + (uint64_t)min(e0 + l_row + 32u * (i - 4u), nrows - 1u) * ncols) + l_c;
        const uint32_t c_end = ncols > 4u * l_c ? (ncols - 4u * l_c + KS - 1u) / KS : 0u;   // steps in which this lane has columns
        auto load = [&](uint32_t ks) {
            if (ks < c_end) {
#pragma unroll
                for (uint32_t i = 0; i < 6; i++) va[i] = __ldg(src[i] + ks * (KS / 4u));
            } else {
#pragma unroll
                for (uint32_t i = 0; i < 6; i++) va[i] = make_float4(0.f, 0.f, 0.f, 0.f);
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
        // sums: this thread's token (a lane of tensor memory) and 16 experts
        float acc[16];
#pragma unroll
        for (int i = 0; i < 16; i++) acc[i] = 0.f;
        const uint32_t e_addr = tmem + ((32u * (warp & 3u)) << 16) + 16u * (warp >> 2);
        auto fold = [&](uint32_t which) {
            tc_fence_after();
            const uint32_t at = e_addr + which * 4u * BN;
#pragma unroll
            for (uint32_t h = 0; h < 16u; h += 8u) {
                uint32_t u[8], v[8], w[8];     // the sums of the large products, the small ones, the smallest
                tmem_ld8(at + h, u), tmem_ld8(at + BN + h, v), tmem_ld8(at + 2u * BN + h, w);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 8; i++) acc[h + i] += __uint_as_float(u[i]) + (__uint_as_float(v[i]) + __uint_as_float(w[i]));
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[which]);
        };
        load(0);
        uint32_t b = 0, ph = 1;
        for (uint32_t ks = 0; ks < nk; ks++) {
            uint8_t *const buf = smem_raw + b * BUF;
            if (ks >= NBUF) wait(&empty[b], ph);                               // step ks - 3 has read its operands
            if (ks >= 4u && (ks & 1u) == 0) fold(((ks - 4u) >> 1) & 1u);        // ... and completed 128 h
#pragma unroll
            for (uint32_t i = 0; i < 4; i++) split(va[i], buf + l_off + 4096u * i, A_PLANE);
#pragma unroll
            for (uint32_t i = 0; i < 2; i++) split(va[4 + i], buf + 3u * A_PLANE + l_off + 4096u * i, B_PLANE);
            if (ks + 1u < nk) load(ks + 1u);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[b]);
            if (++b == NBUF) b = 0, ph ^= 1u;
        }
        for (uint32_t i = nk >= 4u ? nk / 2u - 2u : 0u; i < nk / 2u; i++) {      // the last two accumulators
            wait(&empty[(2u * i + 1u) % NBUF], ((2u * i + 1u) / NBUF) & 1u);
            fold(i & 1u);
        }
        const uint32_t t = t0 + 32u * (warp & 3u) + lane, c0 = e0 + 16u * (warp >> 2);
        if (t < n_tok) {
            float *y = Y + (uint64_t)t * nrows + c0;
            if ((nrows & 3u) == 0 && c0 + 16u <= nrows) {
#pragma unroll
                for (int i = 0; i < 16; i += 4)
                    *reinterpret_cast<float4 *>(y + i) = make_float4(scale * acc[i], scale * acc[i + 1], scale * acc[i + 2], scale * acc[i + 3]);
            } else {
#pragma unroll
                for (int i = 0; i < 16; i++)
                    if (c0 + i < nrows) y[i] = scale * acc[i];
            }
            float z = 0.f;
#pragma unroll
            for (int i = 0; i < 16; i++) z = fmaf(acc[i], 0.f, z);
            if (z != 0.f) plain_logits(W, nrows, ncols, X + (uint64_t)t * ncols, y, c0, scale);   // NaN: one is not finite
        }
    }
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(8u * BN) : "memory");
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
