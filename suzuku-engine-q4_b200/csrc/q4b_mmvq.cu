// The dense product of up to 8 activation rows in 8-bit form: y[t][r] = scale * W[r] . q8(x[t])
// (src/q4.h:913-927, src/q4_mmvq.cu).  Weight types: Q6_K, Q4_K, Q5_K (ggml K-quant super-blocks),
// IQ4_XS and IQ4_NL here; IQ3_S goes through the grouped expert product.
//
// Arithmetic (what makes a row's result independent of the number of rows in the call): the
// activations are quantised per 32 values with d = amax / 127, q = rint(v / d), and the integer sum
// of each half of a group is kept.  A weight row is cut into runs of 16 consecutive values that
// share one scale; each value of a run is a * w + c with integer w.  The lanes of one warp take
// the row's runs round robin and add  dx * (a * dot(w, q) + c * sum16(q))  with explicit fused
// multiply-adds, then the 32 partial sums are added by the xor butterfly.  Every activation row
// goes through exactly these operations, so calls of 1 .. 8 rows give the same bits per row.

namespace mv {

constexpr uint32_t MAXK = Q4B_XQ_MAXLEN;

// ------------------------------------------------------------------ activations
// An integer of magnitude below 2^22 on top of the bits of 1.5 * 2^23, and back to a float: additions at full rate, where
// the conversion instructions run at a quarter of it.
constexpr int BIAS_I = 0x4B400000;
constexpr float BIAS_F = 12582912.f;
__device__ __forceinline__ float unbias(int v) { return __fadd_rn(__int_as_float(v), -BIAS_F); }

// Eight lanes hold a group of 32 values, four each; every lane of the warp calls (src/q4_mmvq.cu:36-57: q = rint(v / d)
// with d = amax / 127, a division and not a product with 127 / amax).  The quotient is taken as a product with the
// reciprocal, which is within 1e-4 of it; only where that is not enough to round (or d has no reciprocal) is it divided.
// Returns the four q; ds: d and the integer sum of this half of the group as a float (at most 2032: exact), which the
// product reads together.
__device__ __forceinline__ uint32_t quant4(float4 v, float2 &ds) {
    float a = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, o));
    const float d = __fdiv_rn(a, 127.f), rd = __fdividef(1.f, d);
    const float val[4] = {v.x, v.y, v.z, v.w};
    uint32_t q[4];
    float off = 0.f;
    bool sure = true;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float p = __fmul_rn(val[i], rd), t = __fadd_rn(p, BIAS_F);
        off = fabsf(__fadd_rn(p, -__fadd_rn(t, -BIAS_F)));
        sure = sure && off <= 0.4998f;   // false for a NaN too
        q[i] = __float_as_uint(t);
    }
    if (!sure) {
#pragma unroll
        for (int i = 0; i < 4; i++) q[i] = d > 0.f ? (uint32_t)__float2int_rn(__fdiv_rn(val[i], d)) : 0u;
    }
    const uint32_t w = __byte_perm(__byte_perm(q[0], q[1], 0x0040), __byte_perm(q[2], q[3], 0x0040), 0x5410);
    int s = __dp4a((int)w, 0x01010101, 0);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    ds = make_float2(d, unbias(s + BIAS_I));
    return w;
}
// values 4 i .. 4 i + 3, of which there are 4 n4 (zeros beyond); x is aligned to a float only
__device__ __forceinline__ float4 ld4(const float *x, uint32_t i, uint32_t n4) {
    if (i >= n4) return make_float4(0.f, 0.f, 0.f, 0.f);
    if (((uintptr_t)x & 15u) == 0) return reinterpret_cast<const float4 *>(x)[i];
    return make_float4(x[4 * (size_t)i], x[4 * (size_t)i + 1], x[4 * (size_t)i + 2], x[4 * (size_t)i + 3]);
}
// rows that q4_mmvq_hold keeps between calls, and those of a call whose y overlaps its x
__global__ void quant8d_k(const float *x, uint32_t n4, uint32_t *__restrict__ q, float2 *__restrict__ ds) {
    q4b_pdl_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    float2 v;
    const uint32_t qw = quant4(ld4(x, i, n4), v);
    if (i < n4) q[i] = qw;
    if (i < n4 && (i & 3u) == 0) ds[i >> 2] = v;
}

// ------------------------------------------------------------------ weight runs
struct Run {
    uint32_t w[4];   // 16 weights, one per byte (unsigned 0..63, or signed codebook values)
    float a, c;
};

__device__ __forceinline__ float f16_lo(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)v)); }

// a and c of sub-block j from the first 16 bytes of a Q4_K / Q5_K block (d, dmin, 12 bytes of 6-bit pairs)
__device__ __forceinline__ void k_scales(uint4 h, uint32_t j, Run &R) {
    const uint32_t sh = 8u * (j & 3u), x0 = h.y >> sh, x1 = h.z >> sh, x2 = h.w >> sh;
    const uint32_t sc = j < 4u ? x0 & 63u : (x2 & 15u) | ((x0 >> 2) & 48u);
    const uint32_t mn = j < 4u ? x1 & 63u : ((x2 >> 4) & 15u) | ((x1 >> 2) & 48u);
    R.a = __fmul_rn(f16_lo(h.x), unbias((int)sc + BIAS_I));
    R.c = __fmul_rn(-f16_lo(h.x >> 16), unbias((int)mn + BIAS_I));
}

// 16 bytes from a 2-byte-aligned address, by halves: aligned words and a funnel shift took longer (5120 x 4096 of Q6_K,
// 3 rows: 26 us a call against 17).
__device__ __forceinline__ uint4 ld16_a2(const uint8_t *p) {
    uint4 v;
    v.x = q4b_ld_u32_a2(p), v.y = q4b_ld_u32_a2(p + 4), v.z = q4b_ld_u32_a2(p + 8), v.w = q4b_ld_u32_a2(p + 12);
    return v;
}

// Per type: Raw, what a run reads; load(block, r) and decode(raw, r) for run r of a block.
template <uint32_t TY> struct Fmt;

// Q6_K, 210 bytes: ql[128] | qh[64] | int8 scales[16] | f16 d.  Each half (128 values) is four
// strips of 32; strip s has its low nibbles in ql bytes 32*(s&1).. of the half (upper nibble for
// s >= 2) and its two high bits in bits 2s..2s+1 of the half's 32 qh bytes.  Values are stored + 32.
template <> struct Fmt<14u> {
    static constexpr uint32_t bytes = 210, vals = 256, align = 2;
    static constexpr bool has_c = true;
    struct Raw {
        uint4 l, h;
        uint32_t d;
        int sc;
    };
    __device__ static uint32_t first(uint32_t r) { return 128u * (r >> 3) + 32u * ((r >> 1) & 3u) + 16u * (r & 1u); }
    __device__ static Raw load(const uint8_t *blk, uint32_t r) {
        const uint32_t half = r >> 3, strip = (r >> 1) & 3u, lo = 16u * (r & 1u);
        Raw v;
        v.l = ld16_a2(blk + 64u * half + 32u * (strip & 1u) + lo);
        v.h = ld16_a2(blk + 128u + 32u * half + lo);
        v.d = q4b_ld_u16(blk + 208);
        v.sc = (int8_t)blk[192u + 8u * half + 2u * strip + (r & 1u)];
        return v;
    }
    __device__ static Run decode(const Raw &v, uint32_t r) {
        const uint32_t strip = (r >> 1) & 3u, sl = 4u * (strip >> 1), sh = 2u * strip;
        Run R;
        R.w[0] = ((v.l.x >> sl) & 0x0F0F0F0Fu) | (((v.h.x >> sh) & 0x03030303u) << 4);
        R.w[1] = ((v.l.y >> sl) & 0x0F0F0F0Fu) | (((v.h.y >> sh) & 0x03030303u) << 4);
        R.w[2] = ((v.l.z >> sl) & 0x0F0F0F0Fu) | (((v.h.z >> sh) & 0x03030303u) << 4);
        R.w[3] = ((v.l.w >> sl) & 0x0F0F0F0Fu) | (((v.h.w >> sh) & 0x03030303u) << 4);
        R.a = __fmul_rn(f16_lo(v.d), unbias(v.sc + BIAS_I));
        R.c = __fmul_rn(-32.f, R.a);
        return R;
    }
};
// Q4_K, 144 bytes: f16 d | f16 dmin | scales[12] | qs[128]; sub-blocks 2p, 2p+1 are the low and
// high nibbles of qs bytes 32p..32p+31
template <> struct Fmt<12u> {
    static constexpr uint32_t bytes = 144, vals = 256, align = 16;
    static constexpr bool has_c = true;
    struct Raw {
        uint4 h, v;
    };
    __device__ static uint32_t first(uint32_t r) { return 16u * r; }
    __device__ static Raw load(const uint8_t *blk, uint32_t r) {
        return {*reinterpret_cast<const uint4 *>(blk), *reinterpret_cast<const uint4 *>(blk + 16u + 32u * (r >> 2) + 16u * (r & 1u))};
    }
    __device__ static Run decode(const Raw &x, uint32_t r) {
        const uint32_t sh = 4u * ((r >> 1) & 1u);
        Run R;
        R.w[0] = (x.v.x >> sh) & 0x0F0F0F0Fu, R.w[1] = (x.v.y >> sh) & 0x0F0F0F0Fu;
        R.w[2] = (x.v.z >> sh) & 0x0F0F0F0Fu, R.w[3] = (x.v.w >> sh) & 0x0F0F0F0Fu;
        k_scales(x.h, r >> 1, R);
        return R;
    }
};
// Q5_K, 176 bytes: as Q4_K with qh[32] before qs; bit j of qh byte l is bit 4 of value l of sub-block j
template <> struct Fmt<13u> {
    static constexpr uint32_t bytes = 176, vals = 256, align = 16;
    static constexpr bool has_c = true;
    struct Raw {
        uint4 h, v, t;
    };
    __device__ static uint32_t first(uint32_t r) { return 16u * r; }
    __device__ static Raw load(const uint8_t *blk, uint32_t r) {
        const uint32_t lo = 16u * (r & 1u);
        return {*reinterpret_cast<const uint4 *>(blk), *reinterpret_cast<const uint4 *>(blk + 48u + 32u * (r >> 2) + lo),
                *reinterpret_cast<const uint4 *>(blk + 16u + lo)};
    }
    __device__ static Run decode(const Raw &x, uint32_t r) {
        const uint32_t j = r >> 1, sh = 4u * (j & 1u);
        Run R;
        R.w[0] = ((x.v.x >> sh) & 0x0F0F0F0Fu) | (((x.t.x >> j) & 0x01010101u) << 4);
        R.w[1] = ((x.v.y >> sh) & 0x0F0F0F0Fu) | (((x.t.y >> j) & 0x01010101u) << 4);
        R.w[2] = ((x.v.z >> sh) & 0x0F0F0F0Fu) | (((x.t.z >> j) & 0x01010101u) << 4);
        R.w[3] = ((x.v.w >> sh) & 0x0F0F0F0Fu) | (((x.t.w >> j) & 0x01010101u) << 4);
        k_scales(x.h, j, R);
        return R;
    }
};
// IQ4_XS, 136 bytes: f16 d | u16 scales_h | scales_l[4] | qs[128]; group ib (32 values) = low then
// high nibbles of qs bytes 16 ib .. 16 ib + 15 through the codebook, 6-bit scale - 32
template <> struct Fmt<23u> {
    static constexpr uint32_t bytes = 136, vals = 256, align = 8;
    static constexpr bool has_c = false;
    struct Raw {
        uint2 h, v0, v1;
    };
    __device__ static uint32_t first(uint32_t r) { return 16u * r; }
    __device__ static Raw load(const uint8_t *blk, uint32_t r) {
        const uint2 *q = reinterpret_cast<const uint2 *>(blk + 8u + 16u * (r >> 1));
        return {*reinterpret_cast<const uint2 *>(blk), q[0], q[1]};
    }
    __device__ static Run decode(const Raw &x, uint32_t r) {
        const uint32_t ib = r >> 1, sh = 4u * (r & 1u);
        Run R;
        R.w[0] = iq4_values4((x.v0.x >> sh) & 0x0F0F0F0Fu), R.w[1] = iq4_values4((x.v0.y >> sh) & 0x0F0F0F0Fu);
        R.w[2] = iq4_values4((x.v1.x >> sh) & 0x0F0F0F0Fu), R.w[3] = iq4_values4((x.v1.y >> sh) & 0x0F0F0F0Fu);
        const int ls = (int)(((x.h.y >> (4u * ib)) & 15u) | (((x.h.x >> (16u + 2u * ib)) & 3u) << 4));
        R.a = __fmul_rn(f16_lo(x.h.x), unbias(ls - 32 + BIAS_I));
        R.c = 0.f;
        return R;
    }
};
// IQ4_NL, 18 bytes per 32 values: f16 d | qs[16]
template <> struct Fmt<20u> {
    static constexpr uint32_t bytes = 18, vals = 32, align = 2;
    static constexpr bool has_c = false;
    struct Raw {
        uint4 v;
        uint32_t d;
    };
    __device__ static uint32_t first(uint32_t r) { return 16u * r; }
    __device__ static Raw load(const uint8_t *blk, uint32_t) { return {ld16_a2(blk + 2), q4b_ld_u16(blk)}; }
    __device__ static Run decode(const Raw &x, uint32_t r) {
        const uint32_t sh = 4u * r;
        Run R;
        R.w[0] = iq4_values4((x.v.x >> sh) & 0x0F0F0F0Fu), R.w[1] = iq4_values4((x.v.y >> sh) & 0x0F0F0F0Fu);
        R.w[2] = iq4_values4((x.v.z >> sh) & 0x0F0F0F0Fu), R.w[3] = iq4_values4((x.v.w >> sh) & 0x0F0F0F0Fu);
        R.a = f16_lo(x.d);
        R.c = 0.f;
        return R;
    }
};

// ------------------------------------------------------------------ the product
// One launch a call: a CTA per SM quantises the activation rows into its shared memory (or copies rows that
// quant8d_k has written) and takes a contiguous share of the weight rows, one or two rows a warp and turn.  With one, the
// rows are split evenly over the turns; with two, the last turn takes one a warp if that is enough (34.6 rows an SM and 32
// in a turn: 6 rows of IQ4_NL 12.9 us a call, 11.6 split evenly).
// A call is short (4096 x 2048 of Q4_K: 4.7 MB, 0.7 us of HBM), so what bounds it is the chain: launch, activations,
// weights, sums.  Quantising in a launch of its own costs more than doing it on every SM; activations and the first rows'
// weights are asked into L2 before the wait for the kernel ahead, later rows one turn in advance.
// In the sums a lane's run has the same place r in its block on every trip (32 runs are whole blocks), so shifts and
// addresses do not change but for a constant step, and two weight rows share a trip's activations (with one row the
// reads of shared memory take longer than the instructions: 24 wavefronts a trip of 4 activation rows).
// A trip's weights are loaded while the sums of the one before run.
// Calls in a graph, 4 rows, 4096 x 2048 of Q4_K: 8.4 us for two launches, 6.1 now; 64 x 2048: 8.4 and 4.9.
// Large matrices are bound by issue: 151,936 x 2048 of Q4_K, 2 / 4 / 8 rows 72 / 94 / 127 us (94, 112, 191 with two launches and
// a warp a row; 27 of bytes), of Q6_K 115 / 144 / 214 (117, 152, 227; 39 of bytes); 4 rows of Q4_K: issue slots 74 % busy.
// 512 threads and two rows a warp; 1024 threads and one row where more warps have to cover the loads and the reads of the
// activations are few: 1 or 2 activation rows (4096 x 2048 of Q5_K, 2 rows: 5.5 us a call against 6.2), types of 2-byte
// alignment, which their narrow loads bound (IQ4_NL, 4 rows: 6.9 against 8.0).  4 rows of Q4_K: 6.1 with 512, 6.5 with 1024.
template <uint32_t TY, int NT> constexpr uint32_t dense_threads = Fmt<TY>::align == 2 || NT <= 2 ? 1024u : 512u;
template <uint32_t TY, int NT>
__global__ void __launch_bounds__(dense_threads<TY, NT>, 1) dense_rows_k(const uint8_t *__restrict__ w, const float *x,
                                                                        const int8_t *gq, const float2 *gds,
                                                                        float *__restrict__ y, uint32_t K, uint32_t rows, float scale) {
    constexpr uint32_t THREADS = dense_threads<TY, NT>;
    using F = Fmt<TY>;
    using Raw = typename F::Raw;
    constexpr uint32_t rpb = F::vals / 16u, step = 32u / rpb * F::bytes, NW_MAX = THREADS / 32u, WR = THREADS == 512u ? 2 : 1;
    extern __shared__ __align__(16) uint8_t smem[];
    int8_t *const xq = reinterpret_cast<int8_t *>(smem);
    float2 *const xds = reinterpret_cast<float2 *>(smem + (size_t)NT * K);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t row_bytes = K / F::vals * F::bytes;
    const uint32_t hi = (uint32_t)((uint64_t)rows * (blockIdx.x + 1u) / gridDim.x);
    uint32_t lo = (uint32_t)((uint64_t)rows * blockIdx.x / gridDim.x);
    const uint32_t turns = (hi - lo + NW_MAX * WR - 1u) / (NW_MAX * WR), NW = WR == 1 ? (hi - lo + turns - 1u) / turns : NW_MAX;
    auto ask = [&](uint32_t rr) {
        if (rr >= hi) return;
        const uint32_t n = min(WR, hi - rr) * row_bytes;
        for (uint32_t o = lane * 128u; o < n; o += 4096u) q4b_l2_prefetch(w + (uint64_t)rr * row_bytes + o);
    };
    const uint32_t n4 = NT * K / 4u;
    if (!gq) {
        const uint32_t i = blockIdx.x + gridDim.x * threadIdx.x;   // lines of the rows, spread over the CTAs
        if (i < n4 / 8u) q4b_l2_prefetch(x + 32u * i);
    }
    if (warp < NW) ask(lo + warp * WR);
    q4b_pdl_wait();
    if (gq) {
        for (uint32_t i = threadIdx.x; i < NT * K / 16u; i += THREADS) {
            reinterpret_cast<uint4 *>(xq)[i] = reinterpret_cast<const uint4 *>(gq)[i];
            xds[i] = gds[i];
        }
    } else {
        for (uint32_t i0 = warp * 32u; i0 < n4; i0 += 4u * THREADS) {
            float4 v[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) v[u] = ld4(x, i0 + u * THREADS + lane, n4);
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {
                const uint32_t i = i0 + u * THREADS + lane;
                if (i0 + u * THREADS >= n4) break;
                float2 ds;
                const uint32_t qw = quant4(v[u], ds);
                if (i < n4) reinterpret_cast<uint32_t *>(xq)[i] = qw;
                if (i < n4 && (i & 3u) == 0) xds[i >> 2] = ds;
            }
        }
    }
    __syncthreads();
    const uint32_t r = lane % rpb, b0 = lane / rpb, e0 = b0 * F::vals + F::first(r);
    auto turn = [&](auto n_tag, uint32_t row) {   // n weight rows from row on
        constexpr int N = decltype(n_tag)::value;
        const uint8_t *wp[N];
#pragma unroll
        for (int i = 0; i < N; i++)
            wp[i] = w + (uint64_t)min(row + (uint32_t)i, hi - 1u) * row_bytes + b0 * F::bytes;
        const int8_t *xp = xq + e0;
        const float2 *dp = xds + (e0 >> 4);
        float acc[N][NT] = {};
        Raw raw[N];
        if (lane < K / 16u) {
#pragma unroll
            for (int i = 0; i < N; i++) raw[i] = F::load(wp[i], r);
        }
#pragma unroll 1
        for (uint32_t run = lane; run < K / 16u; run += 32u) {
            Run R[N];
#pragma unroll
            for (int i = 0; i < N; i++) R[i] = F::decode(raw[i], r);
            if (run + 32u < K / 16u) {   // the next trip's weights, while this one's sums run
#pragma unroll
                for (int i = 0; i < N; i++) wp[i] += step, raw[i] = F::load(wp[i], r);
            }
#pragma unroll
            for (int t = 0; t < NT; t++) {
                const int4 xv = *reinterpret_cast<const int4 *>(xp + t * K);
                const float2 ds = dp[t * (K >> 4)];
#pragma unroll
                for (int i = 0; i < N; i++) {
                    // weights below 128 (or signed codebook values): the signed 4-way dot is exact for both
                    int s = __dp4a((int)R[i].w[0], xv.x, BIAS_I);
                    s = __dp4a((int)R[i].w[1], xv.y, s);
                    s = __dp4a((int)R[i].w[2], xv.z, s);
                    s = __dp4a((int)R[i].w[3], xv.w, s);
                    float v = __fmul_rn(R[i].a, unbias(s));
                    if (F::has_c) v = __fmaf_rn(R[i].c, ds.y, v);
                    acc[i][t] = __fmaf_rn(ds.x, v, acc[i][t]);
                }
            }
            xp += 512u, dp += 32u;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < N; i++)
#pragma unroll
            for (int t = 0; t < NT; t++) {
                float a = acc[i][t];
#pragma unroll
                for (int o = 16; o; o >>= 1) a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, o));
                if (lane == 0 && row + i < hi) y[(size_t)t * rows + row + i] = __fmul_rn(scale, a);
            }
    };
    for (; lo < hi; lo += NW * WR) {
        if (warp >= NW) break;
        ask(lo + (NW + warp) * WR);
        if (WR == 1 || hi - lo <= NW) {
            if (lo + warp < hi) turn(std::integral_constant<int, 1>{}, lo + warp);
        } else if (lo + warp * WR < hi) {
            turn(std::integral_constant<int, (int)WR>{}, lo + warp * WR);
        }
    }
}

// scratch of the quantised rows: q [8][MAXK], scale and sum [8][MAXK / 16]
int8_t *g_q = nullptr;
float2 *g_ds = nullptr;
// what the scratch of either kind holds (q4_mmvq_hold lets calls on the same x reuse it)
const float *g_hold = nullptr;
const float *g_cur_x = nullptr;
uint64_t g_cur_k = 0;
uint32_t g_cur_n = 0;
int g_cur_kind = -1;   // 0: rows of the grouped product (IQ3_S), 1: rows of this file's product
int g_mode = 1;        // 0 off, 1 calls of 2..8 rows, 2 calls of 1..8 rows inside a verify scope only
int g_scope = 0;

bool warm() {
    if (g_q) return true;
    const size_t bytes = (size_t)8 * MAXK + (size_t)8 * (MAXK / 16) * sizeof(float2);
    void *p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    g_q = (int8_t *)p;
    g_ds = (float2 *)(g_q + (size_t)8 * MAXK);
    return true;
}
void shutdown() {
    cudaFree(g_q);
    g_q = nullptr;
    g_ds = nullptr;
    g_hold = g_cur_x = nullptr;
    g_cur_kind = -1;
}

template <uint32_t TY, int N> void launch_n(const uint8_t *w, const float *x, bool held, float *y, uint32_t K, uint32_t rows, float scale) {
    const size_t sm = (size_t)N * (K + K / 16u * sizeof(float2));
    const auto k = dense_rows_k<TY, N>;
    if (sm > 48u * 1024u) (void)cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    q4b_launch(k, rows < (uint32_t)g_q4b.n_sm ? rows : (uint32_t)g_q4b.n_sm, dense_threads<TY, N>, sm, g_q4b.stream, w, x,
               held ? (const int8_t *)g_q : nullptr, (const float2 *)g_ds, y, K, rows, scale);
}
template <uint32_t TY>
bool launch(uint32_t n, const uint8_t *w, const float *x, bool held, float *y, uint32_t K, uint32_t rows, float scale) {
    switch (n) {
#define Q4B_MV_CASE(N)                                       \
    case N: launch_n<TY, N>(w, x, held, y, K, rows, scale); break;
        Q4B_MV_CASE(1) Q4B_MV_CASE(2) Q4B_MV_CASE(3) Q4B_MV_CASE(4) Q4B_MV_CASE(5) Q4B_MV_CASE(6) Q4B_MV_CASE(7)
        Q4B_MV_CASE(8)
#undef Q4B_MV_CASE
    default: return false;
    }
    g_q4b_launches.fetch_add(1, std::memory_order_relaxed);
    return q4b_launch_ok("mmvq_dense");
}

bool dense_type(uint32_t ty) { return ty == 14u || ty == 12u || ty == 13u || ty == 23u || ty == 20u; }

// whole blocks and the row alignment the type's loads need (checked before anything is queued)
template <uint32_t TY> bool fits(const uint8_t *w, uint64_t K) {
    return K % Fmt<TY>::vals == 0 && ((uintptr_t)w % Fmt<TY>::align) == 0 &&
           (K / Fmt<TY>::vals * Fmt<TY>::bytes) % Fmt<TY>::align == 0;
}
bool dense_fits(uint32_t ty, const uint8_t *w, uint64_t K) {
    switch (ty) {
    case 14u: return fits<14u>(w, K);
    case 12u: return fits<12u>(w, K);
    case 13u: return fits<13u>(w, K);
    case 23u: return fits<23u>(w, K);
    case 20u: return fits<20u>(w, K);
    default: return false;
    }
}

}  // namespace mv

bool q4b_mmvq_warm() { return mv::warm(); }
void q4b_mmvq_shutdown() { mv::shutdown(); }

extern "C" void q4_mmvq_warm(void) {
    (void)elem::warm();
    (void)mv::warm();
}
// 0 off; 1 calls of 2..8 rows anywhere; 2 calls of 1..8 rows, only between q4_mmvq_verify(1) and
// q4_mmvq_verify(0) (src/q4_mmvq.cu:271-288).  The reference's per-type thresholds inside modes 1
// and 2 (from 3 rows for some types, short Q4_K tensors only) record where its own float kernels
// were faster on its hardware; this library has no float n-row kernels to fall back to and takes
// every covered type at every n of the mode.
extern "C" int q4_mmvq_on(void) { return g_q4b.ok ? mv::g_mode : 0; }
extern "C" void q4_mmvq_set(int v) { mv::g_mode = v < 0 || v > 2 ? 0 : v; }
extern "C" void q4_mmvq_verify(int on) { mv::g_scope = on ? 1 : 0; }
// Between hold(x) and release(), calls on the same x (same width, no more rows) reuse its
// quantisation; the caller promises x is not rewritten inside the scope (src/q4_mmvq.cu:339-349).
extern "C" void q4_mmvq_hold(const float *d_x) {
    mv::g_hold = d_x;
    mv::g_cur_x = nullptr;
}
extern "C" void q4_mmvq_release(void) {
    mv::g_hold = nullptr;
    mv::g_cur_x = nullptr;
}

extern "C" bool q4_mmvq_n(uint32_t ty, const uint8_t *d_w, uint64_t nrows, uint64_t ncols, const float *d_x,
                          float *d_y, float scale, uint32_t n) {
    const int mode = q4_mmvq_on();
    if (!mode || !d_w || !d_x || !d_y || n < 1 || n > 8 || ncols > mv::MAXK || (ncols % 32) || !nrows ||
        nrows > 0x7fffffffull)
        return false;
    if (mode == 2 ? !mv::g_scope : n < 2) return false;
    const bool dense = mv::dense_type(ty);
    const bool held = mv::g_hold && mv::g_hold == d_x && mv::g_cur_x == d_x && mv::g_cur_k == ncols &&
                      mv::g_cur_kind == (dense ? 1 : 0) && (dense ? mv::g_cur_n >= n : mv::g_cur_n == n);
    if (!dense) {
        // IQ3_S: the rows go through the grouped expert product as one "expert" that owns all n rows,
        // quantised like every other activation of that product
        if (!grouped::shape_ok(ty, nrows, ncols) || !elem::g_mv_xq) return false;
        if (!held) {
            if (!q4_mmq_quantize(d_x, nullptr, elem::g_mv_xq, ty, ncols, n)) return false;
            mv::g_cur_x = d_x, mv::g_cur_k = ncols, mv::g_cur_n = n, mv::g_cur_kind = 0;
        }
        if (!q4_mmq_mul_id(d_w, ty, nrows, ncols, 0, 1, elem::g_mv_xq, elem::g_mv_bounds + 2 * n, n, n, d_y, nrows))
            return false;
        return scale == 1.0f || q4_hip_scale(d_y, scale, (uint64_t)n * nrows);
    }
    if (!mv::g_q || !mv::dense_fits(ty, d_w, ncols)) return false;   // q4_mmvq_warm allocates, outside any stream capture
    const uint32_t K = (uint32_t)ncols, R = (uint32_t)nrows;
    // Rows quantised by a launch of their own: those that hold keeps for further calls, and those of a call that writes
    // its results over them (in dense_rows_k a CTA writes y while others may not have read their x yet).
    const bool keep = mv::g_hold && mv::g_hold == d_x;
    const uintptr_t xa = (uintptr_t)d_x, ya = (uintptr_t)d_y;
    const bool apart = ya >= xa + (uint64_t)n * K * sizeof(float) || xa >= ya + (uint64_t)n * R * sizeof(float);
    if ((keep && !held) || (!keep && !apart)) {
        const uint32_t n4 = n * K / 4u;
        q4b_launch(mv::quant8d_k, (n4 + 255u) / 256u, 256, 0, g_q4b.stream, d_x, n4, (uint32_t *)mv::g_q, mv::g_ds);
        g_q4b_launches.fetch_add(1, std::memory_order_relaxed);
        if (!q4b_launch_ok("mmvq_quant")) return false;
        mv::g_cur_x = d_x, mv::g_cur_k = ncols, mv::g_cur_n = n, mv::g_cur_kind = 1;
    }
    const bool own = keep || !apart;
    switch (ty) {
    case 14u: return mv::launch<14u>(n, d_w, d_x, own, d_y, K, R, scale);
    case 12u: return mv::launch<12u>(n, d_w, d_x, own, d_y, K, R, scale);
    case 13u: return mv::launch<13u>(n, d_w, d_x, own, d_y, K, R, scale);
    case 23u: return mv::launch<23u>(n, d_w, d_x, own, d_y, K, R, scale);
    default: return mv::launch<20u>(n, d_w, d_x, own, d_y, K, R, scale);
    }
}
