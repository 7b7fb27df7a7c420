// Grouped IQ4_NL / IQ4_XS x int8 product (arenas in the engine's byte order) for batches and verify windows: the
// streaming form of wide_rows_k (q4b_wide.cu) on rows of 4-bit codes.  Chunks of whole weight rows come through the
// ring by bulk copies; the codes become int8 codebook values by byte permutes, straight into dp4a words or mma
// fragments.  grouped_rows4_k (q4b_grouped.cu) stays for what the copies cannot take: widths that are not a multiple of
// 128, weights or strides off a 16-byte boundary, a number of rows that is not a multiple of 16.
//
// A code word holds weights 4t..4t+3 of its group in the low and 16+4t.. in the high nibbles.  One permute picks four
// neighbouring NIBBLES (both halves of two bytes), so the values come out as 4t, 16+4t, 4t+1, 17+4t | 4t+2, ...; the
// activation words are brought into the same order instead of the weights.  12 instructions per 8 weights; a table in
// shared memory took 16 lookups and 30 instructions per 16.
//
// Bits are those of grouped_rows4_k: the 32 lane sums of a row there are "slots" here (slot s = groups s, s + 32, ...,
// one after the other) and are added in the order of its butterfly, 16 apart first.
//   1 or 2 rows  a lane is a slot; a row of at most 16 (8) groups takes half (a quarter) of a warp
//   more         mma fragments of 16 weight rows x 8 activation rows; warp ks of KS takes slots ks, ks + KS, ... of a
//                unit of 16 weight rows, in bit-reversed order, so that neighbours in time are a butterfly's pairs
namespace rows4 {

using wide::Args;
using wide::Item;

// Eight weights: both nibbles of bytes 0, 1 of x, and of bytes 2, 3.
__device__ __forceinline__ void values8(uint32_t x, uint32_t &a, uint32_t &b) {
    constexpr uint32_t T0 = iq4_value_word(0), T1 = iq4_value_word(4), T2 = iq4_value_word(8), T3 = iq4_value_word(12);
    const uint32_t s = x & 0x77777777u, y = ((x >> 1) & 0x44444444u) | 0x32103210u;   // low three bits; bit 3 picks the half
    a = q4b_prmt(q4b_prmt(T0, T1, s), q4b_prmt(T2, T3, s), y);
    b = q4b_prmt(q4b_prmt(T0, T1, s >> 16), q4b_prmt(T2, T3, s >> 16), y >> 16);
}
// Activation words k and k + 4 of a group in that order.
__device__ __forceinline__ void order8(uint32_t lo, uint32_t hi, uint32_t &a, uint32_t &b) {
    a = q4b_prmt(lo, hi, 0x5140u);
    b = q4b_prmt(lo, hi, 0x7362u);
}
__device__ __forceinline__ float half_bits(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)v)); }
// d * ls of group g of the row at p (shared memory), as grouped_rows4_k forms it
template <uint32_t T> __device__ __forceinline__ float group_scale(const uint8_t *p, uint32_t g) {
    if (T == Q4_T_IQ4_NL) return half_bits(*reinterpret_cast<const uint16_t *>(p + 18u * g));
    const uint2 h = *reinterpret_cast<const uint2 *>(p + (g >> 3) * 136u);   // d, scales_h | scales_l[4]
    const uint32_t ib = g & 7u;
    const int ls = (int)(((h.y >> (4u * ib)) & 15u) | (((h.x >> (16u + 2u * ib)) & 3u) << 4)) - 32;
    return __fmul_rn(half_bits(h.x & 0xffffu), (float)ls);
}
// Code word t of group g
template <uint32_t T> __device__ __forceinline__ uint32_t code_word(const uint8_t *p, uint32_t g, uint32_t t) {
    if (T == Q4_T_IQ4_XS) return *reinterpret_cast<const uint32_t *>(p + (g >> 3) * 136u + 8u + 16u * (g & 7u) + 4u * t);
    const uint8_t *c = p + 18u * g + 2u + 4u * t;
    return *reinterpret_cast<const uint16_t *>(c) | ((uint32_t)*reinterpret_cast<const uint16_t *>(c + 2) << 16);
}
// All four code words and d * ls
template <uint32_t T> __device__ __forceinline__ float group_words(const uint8_t *p, uint32_t g, uint32_t *w) {
    if (T == Q4_T_IQ4_XS) {
        const uint2 *c = reinterpret_cast<const uint2 *>(p + (g >> 3) * 136u + 8u + 16u * (g & 7u));
        const uint2 x = c[0], y = c[1];
        w[0] = x.x, w[1] = x.y, w[2] = y.x, w[3] = y.y;
        return group_scale<T>(p, g);
    }
    // 18 bytes on a 2-byte boundary: five aligned words, shifted where the block starts on one of their boundaries
    const uint8_t *c = p + 18u * g;
    const uint32_t odd = (uint32_t)(uintptr_t)c & 2u;
    const uint32_t *v = reinterpret_cast<const uint32_t *>(c - odd);
    const uint32_t v0 = v[0], v1 = v[1], v2 = v[2], v3 = v[3], v4 = v[4], sh = odd ? 32u : 16u;
    w[0] = __funnelshift_rc(v0, v1, sh), w[1] = __funnelshift_rc(v1, v2, sh);
    w[2] = __funnelshift_rc(v2, v3, sh), w[3] = __funnelshift_rc(v3, v4, sh);
    return half_bits((odd ? v0 >> 16 : v0) & 0xffffu);
}

// LPR: lanes per weight row in the dp4a form (0: the mma form takes every item); P: passes of a warp over a full chunk
// of 16 P (32 / LPR) rows; J: groups per slot at most.
template <uint32_t T, uint32_t LPR, uint32_t P, uint32_t J>
__global__ void __launch_bounds__(wide::NT, 1) rows4_k(const Args a) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t ng = a.cols >> 5, rb = (uint32_t)iq4_row_bytes(T, a.cols), cr = a.ct;   // a.ct: weight rows of a chunk
    const uint32_t g = lane >> 2, t = lane & 3u, KS = 1u << a.ks_log;
    const uint32_t ks = warp & (KS - 1u), slot = warp >> a.ks_log, n_slot = wide::NCW >> a.ks_log;
    uint32_t m_log = 0;                          // slots of a warp in the mma form: up to 8
    while ((KS << m_log) < min(ng, 32u)) m_log++;
    const uint32_t M = 1u << m_log;
    const uint32_t as = wide::act_stride(a.cols), ss = wide::scale_stride(a.cols);
    wide::stream_items(a, smem_raw, [&](const Item &it, uint32_t &ch, auto &acquire, auto &release) {
        const uint8_t *const ab = it.ab, *const sbase = it.sbase;
        auto few = [&](auto nr_tag) {
            constexpr uint32_t NR = decltype(nr_tag)::value, L = LPR ? LPR : 32u, RPP = 32u / L;
            const uint32_t sl = lane & (L - 1u), sub = lane / L;
            uint32_t q[NR][J][8];
            float dx[NR][J];
#pragma unroll
            for (uint32_t i = 0; i < NR; i++)
#pragma unroll
                for (uint32_t j = 0; j < J; j++) {
                    const uint32_t gi = sl + 32u * j;
                    const bool in = gi < ng;
                    const uint4 *qp = reinterpret_cast<const uint4 *>(ab + i * as + (in ? gi : 0u) * 32u);
                    const uint4 lo = qp[0], hi = qp[1];
                    order8(lo.x, hi.x, q[i][j][0], q[i][j][1]), order8(lo.y, hi.y, q[i][j][2], q[i][j][3]);
                    order8(lo.z, hi.z, q[i][j][4], q[i][j][5]), order8(lo.w, hi.w, q[i][j][6], q[i][j][7]);
                    dx[i][j] = in ? *reinterpret_cast<const float *>(sbase + i * ss + gi * 4u) : 0.f;
                }
            for (; ch < it.ch_stop; ch++) {
                const uint8_t *const sg = acquire();
                const uint32_t rows = min(cr, a.w_rows - ch * cr), r0 = warp * (P * RPP);
                if (r0 < rows) {   // rows past a short chunk's end are computed from what lies there and not stored
                    float v[NR][P];
#pragma unroll
                    for (uint32_t i = 0; i < P; i++) {
                        const uint8_t *const rp = sg + (r0 + i * RPP + sub) * rb;
#pragma unroll
                        for (uint32_t h = 0; h < NR; h++) v[h][i] = 0.f;
#pragma unroll
                        for (uint32_t j = 0; j < J; j++) {
                            const uint32_t gi = sl + 32u * j;
                            if (gi < ng) {
                                uint32_t w[4];
                                const float dl = group_words<T>(rp, gi, w);
                                int I[NR];
#pragma unroll
                                for (uint32_t h = 0; h < NR; h++) I[h] = 0;
#pragma unroll
                                for (uint32_t k = 0; k < 4; k++) {
                                    uint32_t x, y;
                                    values8(w[k], x, y);
#pragma unroll
                                    for (uint32_t h = 0; h < NR; h++)
                                        I[h] = __dp4a((int)y, (int)q[h][j][2 * k + 1], __dp4a((int)x, (int)q[h][j][2 * k], I[h]));
                                }
#pragma unroll
                                for (uint32_t h = 0; h < NR; h++) v[h][i] = fmaf(__fmul_rn(dl, dx[h][j]), (float)I[h], v[h][i]);
                            }
                        }
                    }
                    // the butterfly over a row's lanes; its first steps trade passes between lanes instead of keeping copies
                    const uint32_t pass = P == 4u ? ((sl / (L / 2u)) | (((sl / (L / 4u)) & 1u) << 1)) : sl / (L / 2u);
                    const uint32_t row = r0 + pass * RPP + sub;
                    float *const o = it.out + ch * cr + row;
#pragma unroll
                    for (uint32_t h = 0; h < NR; h++) {
                        const bool up = sl & (L / 2u);
                        float z = up ? v[h][1] : v[h][0];
                        z += __shfl_xor_sync(0xffffffffu, up ? v[h][0] : v[h][1], L / 2u);
                        if (P == 4u) {
                            float y = up ? v[h][3 % P] : v[h][2 % P];
                            y += __shfl_xor_sync(0xffffffffu, up ? v[h][2 % P] : v[h][3 % P], L / 2u);
                            const bool up2 = sl & (L / 4u);
                            const float keep = up2 ? y : z, give = up2 ? z : y;
                            z = keep + __shfl_xor_sync(0xffffffffu, give, L / 4u);
                        }
#pragma unroll
                        for (uint32_t x = L / (P == 4u ? 8u : 4u); x; x >>= 1) z += __shfl_xor_sync(0xffffffffu, z, x);
                        if ((sl & (L / P - 1u)) == 0 && row < rows) o[h * a.ld_dst] = z;
                    }
                }
                release();
            }
        };
        auto many = [&](auto nt_tag) {
            constexpr int NTL = decltype(nt_tag)::value;   // fragments of 8 activation rows: 1 or 2
            const uint8_t *const x0 = ab + g * as + 4u * t;
            const uint8_t *const s0 = sbase + 2u * t * ss;
            for (; ch < it.ch_stop; ch++) {
                const uint8_t *const sg = acquire();
                const uint32_t un = min(cr, a.w_rows - ch * cr) >> 4;
                for (uint32_t u = slot; u < un; u += n_slot) {
                    const uint8_t *const w0 = sg + (u * 16u + g) * rb, *const w1 = w0 + 8u * rb;
                    float lv0[NTL][4], lv1[NTL][4], lv2[NTL][4], sum[NTL][4];
#pragma unroll
                    for (int j = 0; j < NTL; j++)
#pragma unroll
                        for (int o = 0; o < 4; o++) lv0[j][o] = lv1[j][o] = lv2[j][o] = 0.f;
#pragma unroll 1
                    for (uint32_t i = 0; i < M; i++) {
                        const uint32_t m = __brev(i) >> (32u - m_log) & (M - 1u), s = ks + KS * (m_log ? m : 0u);
#pragma unroll
                        for (int j = 0; j < NTL; j++)
#pragma unroll
                            for (int o = 0; o < 4; o++) sum[j][o] = 0.f;
                        for (uint32_t gi = s; gi < ng; gi += 32u) {
                            uint32_t a0, a1, a2, a3;
                            values8(code_word<T>(w0, gi, t), a0, a2);
                            values8(code_word<T>(w1, gi, t), a1, a3);
                            const float dl0 = group_scale<T>(w0, gi), dl1 = group_scale<T>(w1, gi);
#pragma unroll
                            for (int j = 0; j < NTL; j++) {
                                const uint8_t *const xp = x0 + j * 8u * as + gi * 32u;
                                uint32_t b0, b1;
                                order8(*reinterpret_cast<const uint32_t *>(xp), *reinterpret_cast<const uint32_t *>(xp + 16), b0, b1);
                                const float d0 = *reinterpret_cast<const float *>(s0 + j * 8u * ss + gi * 4u);
                                const float d1 = *reinterpret_cast<const float *>(s0 + (j * 8u + 1u) * ss + gi * 4u);
                                int c[4];
                                wide::mma_s8(c, a0, a1, a2, a3, b0, b1);
#pragma unroll
                                for (int o = 0; o < 4; o++)
                                    sum[j][o] = fmaf(__fmul_rn(o < 2 ? dl0 : dl1, (o & 1) ? d1 : d0),
                                                     __int_as_float(c[o]) - wide::MMA_BIAS, sum[j][o]);
                            }
                        }
#pragma unroll
                        for (int j = 0; j < NTL; j++)
#pragma unroll
                            for (int o = 0; o < 4; o++) {   // a binary tree over up to eight slots
                                float x = sum[j][o];
                                if ((i & 1u) == 0) lv0[j][o] = x;
                                else {
                                    x = lv0[j][o] + x;
                                    if ((i & 2u) == 0) lv1[j][o] = x;
                                    else {
                                        x = lv1[j][o] + x;
                                        if ((i & 4u) == 0) lv2[j][o] = x;
                                        else x = lv2[j][o] + x;
                                    }
                                }
                                sum[j][o] = x;
                            }
                    }
                    if (KS > 1u) {   // the warps of the unit meet (one unit a chunk and warp), one fragment after the other
                        const uint32_t bar_n = 32u << a.ks_log, rw = slot * (KS - 1u);
#pragma unroll
                        for (int j = 0; j < NTL; j++) {
                            if (ks) *reinterpret_cast<float4 *>(it.red[rw + ks - 1u][lane]) =
                                make_float4(sum[j][0], sum[j][1], sum[j][2], sum[j][3]);
                            asm volatile("bar.sync %0, %1;" ::"r"(1u + slot), "r"(bar_n) : "memory");
                            if (ks == 0) {
                                auto part = [&](uint32_t i, int o) { return it.red[rw + i - 1u][lane][o]; };
#pragma unroll
                                for (int o = 0; o < 4; o++) {
                                    if (KS == 2u) sum[j][o] += part(1, o);
                                    else if (KS == 4u) sum[j][o] = (sum[j][o] + part(2, o)) + (part(1, o) + part(3, o));
                                    else
                                        sum[j][o] = ((sum[j][o] + part(4, o)) + (part(2, o) + part(6, o))) +
                                                    ((part(1, o) + part(5, o)) + (part(3, o) + part(7, o)));
                                }
                            }
                            asm volatile("bar.sync %0, %1;" ::"r"(1u + slot), "r"(bar_n) : "memory");
                        }
                        if (ks) break;
                    }
                    float *const o0 = it.out + ch * cr + u * 16u + g;
#pragma unroll
                    for (int j = 0; j < NTL; j++)
#pragma unroll
                        for (uint32_t i = 0; i < 2; i++) {
                            const uint32_t r = 8u * j + 2u * t + i;
                            if (r < it.nr) {
                                o0[(uint64_t)r * a.ld_dst] = sum[j][i];
                                o0[(uint64_t)r * a.ld_dst + 8u] = sum[j][2 + i];
                            }
                        }
                }
                release();
            }
        };
        if (LPR != 0 && it.nr == 1u) few(std::integral_constant<uint32_t, 1>{});
        else if (LPR != 0 && it.nr == 2u) few(std::integral_constant<uint32_t, 2>{});
        else if (it.nr <= 8u) many(std::integral_constant<int, 1>{});
        else many(std::integral_constant<int, 2>{});
    });
}

// ---- host side ----
static bool g_ready = false;
template <uint32_t T> static bool warm_type() {
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    const int n = (int)wide::SMEM_MAX;
    return cudaFuncSetAttribute(rows4_k<T, 8, 2, 1>, attr, n) == cudaSuccess &&
           cudaFuncSetAttribute(rows4_k<T, 16, 4, 1>, attr, n) == cudaSuccess &&
           cudaFuncSetAttribute(rows4_k<T, 32, 4, 1>, attr, n) == cudaSuccess &&
           cudaFuncSetAttribute(rows4_k<T, 32, 2, 2>, attr, n) == cudaSuccess &&
           cudaFuncSetAttribute(rows4_k<T, 0, 2, 1>, attr, n) == cudaSuccess;
}
bool warm() {
    g_ready = warm_type<Q4_T_IQ4_NL>() && warm_type<Q4_T_IQ4_XS>();
    if (!g_ready) cudaGetLastError();
    return g_ready;
}
template <uint32_t T> static void launch_type(const Args &a, uint32_t ng, size_t sm) {
    if (ng <= 8u) q4b_launch(rows4_k<T, 8, 2, 1>, g_q4b.n_sm, wide::NT, sm, g_q4b.stream, a);
    else if (ng <= 16u) q4b_launch(rows4_k<T, 16, 4, 1>, g_q4b.n_sm, wide::NT, sm, g_q4b.stream, a);
    else if (ng <= 32u) q4b_launch(rows4_k<T, 32, 4, 1>, g_q4b.n_sm, wide::NT, sm, g_q4b.stream, a);
    else if (ng <= 64u) q4b_launch(rows4_k<T, 32, 2, 2>, g_q4b.n_sm, wide::NT, sm, g_q4b.stream, a);
    else q4b_launch(rows4_k<T, 0, 2, 1>, g_q4b.n_sm, wide::NT, sm, g_q4b.stream, a);
}
// false: not this kernel's shape, nothing queued.  Chunks of about 36 KB whatever the width; a row of more than 2048
// columns goes through the fragments whatever its entry's rows (its activation words would not fit a lane's registers).
bool launch(uint32_t type, Args a) {
    const uint32_t ng = a.cols >> 5;
    const uint64_t rb = iq4_row_bytes(type, a.cols);
    if (!g_ready || (a.cols % 128u) || ng > 128u || (a.w_rows % 16u) || a.n_entries > wide::MAX_ENTRIES ||
        (((uintptr_t)a.w | a.expert_stride) & 15u))
        return false;
    const uint32_t p = ng <= 8u || ng > 32u ? 2u : 4u, rpp = ng <= 8u ? 4u : ng <= 16u ? 2u : 1u;
    for (a.ct = 16u * p * rpp;; a.ct /= 2u) {
        const uint32_t units = a.ct / 16u;
        a.ks_log = 0;
        while ((units << (a.ks_log + 1u)) <= wide::NCW && a.ks_log < 3u) a.ks_log++;
        a.chunk_bytes = (uint32_t)(a.ct * rb);
        a.n_stage = wide::MAX_STAGE;
        while (a.n_stage >= 2u && wide::smem_bytes(a.cols, a.chunk_bytes, a.n_stage) > wide::SMEM_MAX) a.n_stage--;
        if (a.n_stage >= 2u || ng <= 64u || a.ct == 16u) break;
    }
    if (a.n_stage < 2u) return false;
    a.cpe = (a.w_rows + a.ct - 1u) / a.ct;
    a.last_bytes = (uint32_t)((a.w_rows - (a.cpe - 1u) * a.ct) * rb);
    const size_t sm = wide::smem_bytes(a.cols, a.chunk_bytes, a.n_stage);
    if (type == Q4_T_IQ4_NL) launch_type<Q4_T_IQ4_NL>(a, ng, sm);
    else launch_type<Q4_T_IQ4_XS>(a, ng, sm);
    return true;
}

}  // namespace rows4
