// Grouped IQ3_S x int8 product for few activation rows per expert on the wide form of an arena
// (q4b_tile.cuh): batched decode, verify windows, expert-parallel shards.  Same work as grouped_few_k
// (q4b_few.cu), which stays for tiled arenas without a wide copy.
//
// A persistent kernel, one CTA of 16 warps per SM.  Work is cut into items (an
// expert, a block of up to 16 of its rows) and chunks (up to 64 tiles of its weights); the CTAs take
// contiguous shares of the chunk list by estimated cost.  A ring of chunks is kept in flight with 1-D bulk
// copies, which also bring an item's activation rows (8-bit values and scales) into one of
// two buffers with its first chunk, so that a change of experts costs no round trip to memory.
//
// Two inner forms, chosen per item by its rows:
//   1 or 2 rows  a lane owns a tile's groups 2l, 2l+1 (block l/4), its 64 activation bytes a row live
//                in registers, dp4a; the sums of a warp's tiles are reduced together, so four tiles
//                cost six shuffles a row instead of twenty
//   3..16 rows   integer mma m16n8k32 (16 weight rows x 8 activation rows x one 32-group): the weight
//                words of lane (g, t) ARE the A fragment after one AND-OR per half, the activations are
//                the B fragment as they lie in shared memory.  Warps split a unit of 16 weight rows
//                along k when a chunk has fewer than 16 units.
// Both form the exact integer dot of every 32-group (times 8) and then the expression and the order of
// additions of grouped_rows_k (pairs of groups, blocks of four pairs, blocks pairwise), so for 1, 2, 4 or 8
// super-blocks a row the result is that kernel's, bit for bit.
//
// What bounds it: with 1 or 2 rows an entry start-up and HBM (1088 bytes a tile: 90 us for 370 experts' gate/up against 64
// of bytes), from 3 rows on instruction issue.  64 tokens of 11 picks (369 experts, 1.9 rows): 137 warp instructions a
// tile, issue slots 63 % busy, DRAM at 59 % of its peak, 88.6 us under the profiler.  The tiled form took 247 with 1.7 rows.
#include "q4b_tile.cuh"

#include <type_traits>

const uint8_t *q4b_wide_of(const void *p);

namespace wide {

constexpr uint32_t NCW = 16;                     // warps
constexpr uint32_t NT = 32 * NCW;
constexpr uint32_t MAX_ENTRIES = 1024;
constexpr uint32_t RBLK = 16;                    // activation rows of an item at most
constexpr uint32_t MAX_STAGE = 8;
constexpr uint32_t WAIT_LIMIT = 1u << 21;        // tries before a wait gives up ...
constexpr unsigned long long WAIT_NS = 500000000ull;   // ... or half a second, whichever comes first
constexpr uint32_t ERR_WIDE = 0x1000u;

struct Smem {
    unsigned long long full[MAX_STAGE], act_full[2];
    uint32_t done[MAX_STAGE];                    // warps that are through with a stage's chunk
    // where the two streams stand (entry of the live list, block of rows): chunks, activation rows
    uint32_t p_li, p_blk, p_ch, p_nb, x_li, x_blk, x_item;
    uint32_t i_row[2], i_nr[2], i_nb[2];         // item in an activation buffer: first row, rows, blocks of its entry
    const uint8_t *p_mat;
    alignas(16) float red[NCW - 2][32][4];                // partial sums of warps that share a unit (all but one of each unit)
    uint32_t live[MAX_ENTRIES];                  // entries with rows
    uint32_t cost[MAX_ENTRIES + 1];              // cost of everything before entry i of that list
    uint32_t wl[NCW], wc[NCW];                   // per-warp sums of the scan
};

struct Args {
    const uint8_t *w;            // wide form of expert 0's matrix
    uint64_t expert_stride;      // in wide bytes
    const int32_t *act;
    const uint32_t *n_act;
    uint32_t n_entries;
    const int32_t *bounds;
    const int8_t *xq;
    const float *xd;
    uint32_t cols, w_rows;
    float *dst;
    uint64_t ld_dst;
    uint32_t *err;
    uint32_t ct;                 // tiles per chunk (whole units)
    uint32_t n_stage;            // chunks in the ring
    uint32_t ks_log;             // log2 of the warps per unit of 16 weight rows in the mma form
    uint32_t cpe;                // chunks of a matrix
    uint32_t chunk_bytes, last_bytes;
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, uint32_t parity, uint32_t limit, uint32_t *err) {
    const uint32_t a = smem_u32(bar);
    unsigned long long t0 = 0;
    for (uint32_t i = 0; i < limit; i++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
        if ((i & 1023u) == 1023u) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
            if (t0 == 0) t0 = t;
            else if (t - t0 > WAIT_NS) break;
        }
    }
    atomicOr(err, ERR_WIDE);
    return false;
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, unsigned long long *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
// D = A (16 x 32, int8) * B (32 x 8, int8) in int32, on top of the bits of the float 1.5 * 2^23: the sum's
// magnitude is below 2^22, so the bits read as a float are MMA_BIAS + the sum
constexpr float MMA_BIAS = 12582912.f;
__device__ __forceinline__ void mma_s8(int *c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%10, %10, %10, %10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(__float_as_int(MMA_BIAS)));
}
// 1 + 2 s of the nibble s in the low bits, by way of the float 2^23 + s; and -MMA_BIAS times it
__device__ __forceinline__ float sub_scale(uint32_t s) {
    return __fmaf_rn(2.f, __uint_as_float((s & 15u) | 0x4b000000u), -16777215.f);
}
// The same for the nibble at bit `at` (a constant, at most 16): the float is 2^23 + s 2^at.
__device__ __forceinline__ void sub_scale(uint32_t s, uint32_t at, float &l, float &k) {
    const float x = __uint_as_float((s & (15u << at)) | 0x4b000000u);
    l = __fmaf_rn(x, 2.f / (float)(1u << at), 1.f - 16777216.f / (float)(1u << at));
    k = __fmul_rn(l, -MMA_BIAS);
}
// smem strides of an activation row and of its scales (padding against bank conflicts)
__host__ __device__ inline uint32_t act_stride(uint32_t cols) { return cols + 32u; }
__host__ __device__ inline uint32_t scale_stride(uint32_t cols) { return (cols >> 5) * 4u + 16u; }
__host__ __device__ inline uint32_t act_bytes(uint32_t cols) {
    return (RBLK * (act_stride(cols) + scale_stride(cols)) + 127u) & ~127u;
}
__host__ __device__ inline uint32_t smem_bytes(uint32_t cols, uint32_t chunk_bytes, uint32_t n_stage) {
    return (uint32_t)((sizeof(Smem) + 127u) & ~127u) + 2u * act_bytes(cols) + n_stage * chunk_bytes;
}
// Relative cost of a chunk for a block of rows: the stream of its bytes until the rows' own work exceeds it
// (370 experts, gate/up, events around one call: 90 us with 1 row, 92 with 2, 115 with 8, 152 with 16).
__device__ __forceinline__ uint32_t block_cost(uint32_t rows) {
    return rows <= 2u ? 7u + rows : rows <= 8u ? 12u : 17u;
}
// An entry's rows are split into blocks of RBLK, the rest in the last (512 experts of 17 / 24 rows, gate/up, under the profiler:
// 279 / 340 us; as 9 and 8, and twice 12 rows, 341 / 395: two fragments each, half empty).
__device__ __forceinline__ uint32_t row_blocks(uint32_t rows) { return (rows + RBLK - 1u) / RBLK; }
__device__ __forceinline__ uint32_t entry_cost(uint32_t rows, uint32_t cpe) {
    const uint32_t nb = row_blocks(rows);
    return cpe * ((nb - 1u) * block_cost(RBLK) + block_cost(rows - (nb - 1u) * RBLK));
}

// One item as the body of a kernel sees it: rows, where its results go, its activation rows and their scales in shared
// memory; the chunks [ch, ch_stop) of its weights are taken one after the other (acquire, release).
struct Item {
    uint32_t nr;
    float *out;
    const uint8_t *ab, *sbase;
    uint32_t ch_stop;
    float (*red)[32][4];
};
// Streams this CTA's share of the (item, chunk) list through the ring and hands every item to body(item, ch, acquire,
// release); the body advances ch to ch_stop.
template <typename Body> __device__ __forceinline__ void stream_items(const Args &a, uint8_t *smem_raw, const Body &body) {
    Smem &s = *reinterpret_cast<Smem *>(smem_raw);
    uint8_t *const actb = smem_raw + ((sizeof(Smem) + 127u) & ~127u);
    const uint32_t act_sz = act_bytes(a.cols), sc_off = RBLK * act_stride(a.cols);
    uint8_t *const stage = actb + 2u * act_sz;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t cpe = a.cpe;
    if (tid == 0) {
        for (uint32_t i = 0; i < a.n_stage; i++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&s.full[i])), "r"(1u));
            s.done[i] = 0;
        }
        for (uint32_t i = 0; i < 2; i++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&s.act_full[i])), "r"(1u));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    q4b_pdl_wait();
    const uint32_t n_ent = a.n_act ? min(*a.n_act, a.n_entries) : a.n_entries;
    // ---- the live entries and the prefix of their costs: a thread takes two neighbouring entries ----
    uint32_t n_live, total_cost;
    {
        uint32_t r[2], lv = 0, cs = 0;
#pragma unroll
        for (uint32_t h = 0; h < 2; h++) {
            const uint32_t e = 2u * tid + h;
            const int32_t nr = e < n_ent ? a.bounds[e + 1] - a.bounds[e] : 0;
            r[h] = nr > 0 ? (uint32_t)nr : 0u;
            if (r[h]) {
                lv++;
                cs += entry_cost(r[h], cpe);
            }
        }
        uint32_t il = lv, ic = cs;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t tl = __shfl_up_sync(0xffffffffu, il, o), tc = __shfl_up_sync(0xffffffffu, ic, o);
            if (lane >= (uint32_t)o) il += tl, ic += tc;
        }
        if (lane == 31u) s.wl[warp] = il, s.wc[warp] = ic;
        __syncthreads();
        uint32_t pl = il - lv, pc = ic - cs;
        n_live = 0, total_cost = 0;
#pragma unroll
        for (uint32_t i = 0; i < NCW; i++) {
            if (i < warp) pl += s.wl[i], pc += s.wc[i];
            n_live += s.wl[i], total_cost += s.wc[i];
        }
#pragma unroll
        for (uint32_t h = 0; h < 2; h++)
            if (r[h] && pl < MAX_ENTRIES) {
                s.live[pl] = 2u * tid + h;
                s.cost[pl] = pc;
                pl++;
                pc += entry_cost(r[h], cpe);
            }
        if (tid == 0) s.cost[n_live] = total_cost;
    }
    __syncthreads();
    if (n_live == 0) return;
    // first chunk (entry, chunk of its nb * cpe) whose start cost is >= target
    auto locate = [&](uint64_t target, uint32_t &ent, uint32_t &idx) {
        if (target >= total_cost) {
            ent = n_live, idx = 0;
            return;
        }
        uint32_t lo = 0, hi = n_live;
        while (hi - lo > 1u) {
            const uint32_t mid = (lo + hi) >> 1;
            if (s.cost[mid] <= target) lo = mid;
            else hi = mid;
        }
        const uint32_t e = s.live[lo], rows = (uint32_t)(a.bounds[e + 1] - a.bounds[e]);
        const uint32_t nb = row_blocks(rows), n = nb * cpe, n_full = (nb - 1u) * cpe;      // chunks, and those of whole blocks
        const uint32_t off = (uint32_t)target - s.cost[lo], full = block_cost(RBLK), last = block_cost(rows - (nb - 1u) * RBLK);
        const uint32_t w = off <= n_full * full ? (off + full - 1u) / full : n_full + (off - n_full * full + last - 1u) / last;
        ent = w >= n ? lo + 1u : lo;
        idx = w >= n ? 0u : w;
    };
    uint32_t li, ix, li_end, ix_end;
    locate((uint64_t)total_cost * blockIdx.x / gridDim.x, li, ix);
    locate((uint64_t)total_cost * (blockIdx.x + 1ull) / gridDim.x, li_end, ix_end);

    // ---- the streams ----
    // The warp that is last through a chunk refills its stage with the next chunk of this CTA's share, and the one that
    // is last through an item's last chunk brings the activation rows of the item after the next into the buffer
    // that has become free (one lane; refills come in order, because a warp leaves chunk k + 1 only after it has
    // refilled behind chunk k).
    const uint32_t blk_end = ix_end / cpe, ch_end = ix_end - blk_end * cpe, chunk_bytes = a.chunk_bytes;
    auto enter = [&](uint32_t pl) {   // the entry whose chunks come next (behind the copy before: its loads take a while)
        const uint32_t e = s.live[pl];
        const int32_t b0 = a.bounds[e], b1 = a.bounds[e + 1], slot = a.act ? a.act[e] : (int32_t)e;
        s.p_nb = row_blocks((uint32_t)(b1 - b0));
        s.p_mat = a.w + (uint64_t)slot * a.expert_stride;
    };
    auto refill = [&](uint32_t st) {
        uint32_t pl = s.p_li, pb = s.p_blk, pc = s.p_ch;
        if (pl == li_end && pb == blk_end && pc == ch_end) return;
        const uint32_t bytes = pc + 1u == cpe ? a.last_bytes : chunk_bytes;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&s.full[st])), "r"(bytes) : "memory");
        bulk_g2s(stage + st * chunk_bytes, s.p_mat + (uint64_t)pc * chunk_bytes, bytes, &s.full[st]);
        if (++pc == cpe) {
            pc = 0;
            if (++pb == s.p_nb) {
                pb = 0;
                if (++pl < n_live) enter(pl);
            }
        }
        s.p_li = pl, s.p_blk = pb, s.p_ch = pc;
    };
    auto refill_rows = [&]() {
        uint32_t xl = s.x_li, xb = s.x_blk;
        if (xl > li_end || (xl == li_end && (xb > blk_end || (xb == blk_end && ch_end == 0)))) return;   // past the share
        const uint32_t e = s.live[xl], buf = s.x_item & 1u, sb = (a.cols >> 5) * 4u;
        const int32_t b0 = a.bounds[e], b1 = a.bounds[e + 1];
        const uint32_t rows = (uint32_t)(b1 - b0);
        const uint32_t nb = row_blocks(rows), nr = min(RBLK, rows - xb * RBLK);
        const uint64_t r0 = (uint64_t)b0 + xb * RBLK;
        uint8_t *const ab = actb + buf * act_sz;
        s.i_row[buf] = (uint32_t)r0, s.i_nr[buf] = nr, s.i_nb[buf] = nb;   // seen by who waits for the copies
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&s.act_full[buf])),
                     "r"(nr * (a.cols + sb))
                     : "memory");
        for (uint32_t i = 0; i < nr; i++) {
            bulk_g2s(ab + i * act_stride(a.cols), a.xq + (r0 + i) * a.cols, a.cols, &s.act_full[buf]);
            bulk_g2s(ab + sc_off + i * scale_stride(a.cols), a.xd + (r0 + i) * (a.cols >> 5), sb, &s.act_full[buf]);
        }
        if (++xb == nb) xb = 0, xl++;
        s.x_li = xl, s.x_blk = xb, s.x_item++;
    };
    if (tid == 0 && (li != li_end || ix != ix_end)) {
        s.p_li = s.x_li = li, s.p_blk = s.x_blk = ix / cpe, s.p_ch = ix % cpe, s.x_item = 0;
        enter(li);
        refill_rows();
        for (uint32_t i = 0; i < a.n_stage; i++) refill(i);
        refill_rows();
    }

    // ---- the warps ----
    uint32_t st = 0, ph = 0, item = 0, limit = WAIT_LIMIT, blk = ix / cpe, ch = ix - blk * cpe;
    // one item: a chunk after the other
    while (li != li_end || blk != blk_end || ch != ch_end) {
        const uint32_t buf = item & 1u;
        const uint8_t *const ab = actb + buf * act_sz, *const sbase = ab + sc_off;
        if (!mbar_wait(&s.act_full[buf], (item >> 1) & 1u, limit, a.err)) limit = 1024u;
        const uint32_t nr = s.i_nr[buf], nb = s.i_nb[buf];
        float *const out = a.dst + (uint64_t)s.i_row[buf] * a.ld_dst;
        const uint32_t ch_stop = li == li_end && blk == blk_end ? ch_end : cpe;
        auto acquire = [&]() {
            if (!mbar_wait(&s.full[st], ph, limit, a.err)) limit = 1024u;
            return (const uint8_t *)(stage + st * chunk_bytes);
        };
        auto release = [&]() {
            __syncwarp();
            if (lane == 0) {
                uint32_t n;
                asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(n) : "r"(smem_u32(&s.done[st])) : "memory");
                if (n == NCW - 1u) {
                    s.done[st] = 0;
                    if (ch + 1u == cpe) refill_rows();   // the item's last chunk: its buffer is free
                    refill(st);
                }
            }
            if (++st == a.n_stage) st = 0, ph ^= 1u;
        };
        const Item it = {nr, out, ab, sbase, ch_stop, s.red};
        body(it, ch, acquire, release);
        if (ch_stop != cpe) break;         // the end of this CTA's share
        item++;
        ch = 0, blk++;
        if (blk == nb) blk = 0, li++;
    }
}

// BB: super-blocks per weight row, 1, 2, 4 or 8; 0 = another number (mma form only).  TPW: tiles a warp takes
// from a full chunk in the dp4a form.
template <uint32_t BB, uint32_t TPW>
__global__ void __launch_bounds__(NT, 1) wide_rows_k(const Args a) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, cpe = a.cpe;
    const uint32_t B = BB ? BB : a.cols >> 8, last_tiles = (a.w_rows >> 3) * B - (cpe - 1u) * a.ct;
    const uint32_t rows_per_chunk = a.ct / B * 8u;
    // mma form: lane (g, t) of a fragment; this warp's unit slot and its share of a unit's super-blocks
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint32_t ks = warp & ((1u << a.ks_log) - 1u), slot = warp >> a.ks_log, n_slot = NCW >> a.ks_log;
    const uint32_t b_lo = (B * ks) >> a.ks_log, b_hi = (B * (ks + 1u)) >> a.ks_log;
    stream_items(a, smem_raw, [&](const Item &it, uint32_t &ch, auto &acquire, auto &release) {
        const uint32_t nr = it.nr, ch_stop = it.ch_stop;
        float *const out = it.out;
        const uint8_t *const ab = it.ab, *const sbase = it.sbase;
        auto few = [&](auto nr_tag) {
            constexpr uint32_t NR = decltype(nr_tag)::value, B1 = BB ? BB : 1u, lpr = 4u * B1, rpt = 8u / B1;
            const uint32_t p = lane & 3u, bl = lane >> 2;
            const uint8_t *sg = acquire();
            int q[NR][16];            // this lane's 64 columns of the item's rows
            float dx[NR][2];
            const uint32_t gcol = (bl & (B1 - 1u)) * 8u + 2u * p;
#pragma unroll
            for (uint32_t i = 0; i < NR; i++) {
                const uint4 *qp = reinterpret_cast<const uint4 *>(ab + i * act_stride(a.cols) + gcol * 32u);
#pragma unroll
                for (uint32_t j = 0; j < 4; j++) {
                    const uint4 v = qp[j];
                    q[i][4 * j] = (int)v.x, q[i][4 * j + 1] = (int)v.y;
                    q[i][4 * j + 2] = (int)v.z, q[i][4 * j + 3] = (int)v.w;
                }
                const float2 dv = *reinterpret_cast<const float2 *>(sbase + i * scale_stride(a.cols) + gcol * 4u);
                dx[i][0] = dv.x, dx[i][1] = dv.y;
            }
            const uint32_t t0 = warp * TPW, tl = t0 + (lane & (TPW - 1u));   // this warp's tiles; the one this lane stores
            const bool o1 = lane & 1u, o2 = lane & 2u;
            float *dst = out + (ch * a.ct + tl) * rpt + lane / lpr;
            for (;;) {
                const uint32_t tiles = ch + 1u == cpe ? last_tiles : a.ct;
                if (t0 < tiles) {   // tiles past a short chunk's end are computed from what lies there and not stored
                    const uint8_t *tile = sg + t0 * Q4B_WIDE_BYTES + 8u * lane;
                    const uint8_t *rp = sg + t0 * Q4B_WIDE_BYTES + Q4B_WIDE_PART * (bl >> 1) + 256u + 8u * (bl & 1u);
                    float v[NR][TPW];
#pragma unroll
                    for (uint32_t i = 0; i < TPW; i++) {
                        int a0[NR], a1[NR];
#pragma unroll
                        for (uint32_t h = 0; h < NR; h++) a0[h] = a1[h] = 0;
#pragma unroll
                        for (uint32_t t4 = 0; t4 < 4; t4++) {
                            const uint2 w = *reinterpret_cast<const uint2 *>(tile + i * Q4B_WIDE_BYTES + Q4B_WIDE_PART * t4);
                            const int x0 = (int)q4b_wide_lo(w.x), x1 = (int)q4b_wide_hi(w.x);
                            const int y0 = (int)q4b_wide_lo(w.y), y1 = (int)q4b_wide_hi(w.y);
#pragma unroll
                            for (uint32_t h = 0; h < NR; h++) {
                                a0[h] = __dp4a(x1, q[h][2 * t4 + 1], __dp4a(x0, q[h][2 * t4], a0[h]));
                                a1[h] = __dp4a(y1, q[h][8 + 2 * t4 + 1], __dp4a(y0, q[h][8 + 2 * t4], a1[h]));
                            }
                        }
                        const uint2 rec = *reinterpret_cast<const uint2 *>(rp + i * Q4B_WIDE_BYTES);
                        const float d = __half2float(__ushort_as_half((unsigned short)rec.x)) * 0.125f;   // the dots are 8 w q
                        const uint32_t sc = rec.y >> (8u * p);
                        const float ls0 = sub_scale(sc), ls1 = sub_scale(sc >> 4);
#pragma unroll
                        for (uint32_t h = 0; h < NR; h++)   // dot x sub-scale is below 2^24: exact
                            v[h][i] = __fmul_rn(d, __fmaf_rn((float)a0[h] * ls0, dx[h][0], __fmul_rn((float)a1[h] * ls1, dx[h][1])));
                    }
                    // sums over a weight row's lanes: the first steps trade tiles between lanes instead of
                    // keeping copies (the same pairs are added, in the order of a plain butterfly)
#pragma unroll
                    for (uint32_t h = 0; h < NR; h++) {
                        float z;
                        if (TPW == 4) {
                            float x = o1 ? v[h][1] : v[h][0], y = o1 ? v[h][3 % TPW] : v[h][2 % TPW];
                            x += __shfl_xor_sync(0xffffffffu, o1 ? v[h][0] : v[h][1], 1);
                            y += __shfl_xor_sync(0xffffffffu, o1 ? v[h][2 % TPW] : v[h][3 % TPW], 1);
                            z = o2 ? y : x;
                            z += __shfl_xor_sync(0xffffffffu, o2 ? x : y, 2);
                        } else {
                            z = o1 ? v[h][1] : v[h][0];
                            z += __shfl_xor_sync(0xffffffffu, o1 ? v[h][0] : v[h][1], 1);
                            z += __shfl_xor_sync(0xffffffffu, z, 2);
                        }
                        if (B1 >= 2) z += __shfl_xor_sync(0xffffffffu, z, 4);
                        if (B1 >= 4) z += __shfl_xor_sync(0xffffffffu, z, 8);
                        if (B1 >= 8) z += __shfl_xor_sync(0xffffffffu, z, 16);
                        if ((lane & (lpr - 1u)) < TPW && tl < tiles) dst[h * a.ld_dst] = z;
                    }
                }
                release();
                if (++ch == ch_stop) break;
                dst += a.ct * rpt;
                sg = acquire();
            }
        };
        auto many = [&](auto nt_tag) {
            constexpr int NTL = decltype(nt_tag)::value;   // fragments of 8 activation rows: 1 or 2
            const uint8_t *const x0 = ab + g * act_stride(a.cols) + 8u * t;
            const uint8_t *const s0 = sbase + 2u * t * scale_stride(a.cols), *const s1 = s0 + scale_stride(a.cols);
            for (; ch < ch_stop; ch++) {
                const uint8_t *const sg = acquire();
                const uint32_t un = (ch + 1u == cpe ? last_tiles : a.ct) / (2u * B);
                for (uint32_t u = slot; u < un; u += n_slot) {
                    float sum[NTL][4];
                    // Blocks of the lane's two weight rows, g and g + 8 of the unit.  For B = 1, 2, 4, 8 a row
                    // lies in one tile and both rows start at the same block of theirs.
                    const uint32_t r0b = (u * 16u + g) * B, r1b = r0b + 8u * B;
                    const uint8_t *t0 = sg + (r0b >> 3) * Q4B_WIDE_BYTES, *t1 = sg + (r1b >> 3) * Q4B_WIDE_BYTES;
#pragma unroll 1
                    for (uint32_t b = b_lo; b < b_hi; b++) {
                        uint32_t k0 = (r0b & 7u) + b, k1 = k0;
                        if (BB == 0) {
                            k0 = (r0b + b) & 7u, k1 = (r1b + b) & 7u;
                            t0 = sg + ((r0b + b) >> 3) * Q4B_WIDE_BYTES, t1 = sg + ((r1b + b) >> 3) * Q4B_WIDE_BYTES;
                        }
                        const uint4 *wp0 = reinterpret_cast<const uint4 *>(t0 + Q4B_WIDE_PART * t + k0 * 32u);
                        const uint4 *wp1 = reinterpret_cast<const uint4 *>(t1 + Q4B_WIDE_PART * t + k1 * 32u);
                        const uint4 wa0 = wp0[0], wb0 = wp0[1], wa1 = wp1[0], wb1 = wp1[1];
                        const uint2 rc0 = *reinterpret_cast<const uint2 *>(t0 + Q4B_WIDE_PART * (k0 >> 1) + 256u + 8u * (k0 & 1u));
                        const uint2 rc1 = *reinterpret_cast<const uint2 *>(t1 + Q4B_WIDE_PART * (k1 >> 1) + 256u + 8u * (k1 & 1u));
                        const float d0 = __half2float(__ushort_as_half((unsigned short)rc0.x)) * 0.125f;
                        const float d1 = __half2float(__ushort_as_half((unsigned short)rc1.x)) * 0.125f;
                        const uint32_t rh0 = rc0.y >> 20, rh1 = rc1.y >> 20;
                        const uint8_t *const xb = x0 + b * 256u, *const sb0 = s0 + b * 32u, *const sb1 = s1 + b * 32u;
                        float bs[NTL][4], hold[NTL][4];
#pragma unroll
                        for (uint32_t p = 0; p < 4; p++) {
                            const uint32_t w00 = p == 0 ? wa0.x : p == 1 ? wa0.z : p == 2 ? wb0.x : wb0.z;
                            const uint32_t w01 = p == 0 ? wa0.y : p == 1 ? wa0.w : p == 2 ? wb0.y : wb0.w;
                            const uint32_t w10 = p == 0 ? wa1.x : p == 1 ? wa1.z : p == 2 ? wb1.x : wb1.z;
                            const uint32_t w11 = p == 0 ? wa1.y : p == 1 ? wa1.w : p == 2 ? wb1.y : wb1.w;
                            float l00, l01, l10, l11, k00, k01, k10, k11;   // sub-scales of the two rows' groups, and their biases
                            if (p < 3) sub_scale(rc0.y, 8u * p, l00, k00), sub_scale(rc1.y, 8u * p, l10, k10);
                            else sub_scale(rh0, 4u, l00, k00), sub_scale(rh1, 4u, l10, k10);
                            if (p < 2) sub_scale(rc0.y, 8u * p + 4u, l01, k01), sub_scale(rc1.y, 8u * p + 4u, l11, k11);
                            else sub_scale(rh0, 8u * p - 16u, l01, k01), sub_scale(rh1, 8u * p - 16u, l11, k11);
                            const uint32_t a00 = q4b_wide_lo(w00), a02 = q4b_wide_hi(w00), a01 = q4b_wide_lo(w10), a03 = q4b_wide_hi(w10);
                            const uint32_t e00 = q4b_wide_lo(w01), e02 = q4b_wide_hi(w01), e01 = q4b_wide_lo(w11), e03 = q4b_wide_hi(w11);
#pragma unroll
                            for (int j = 0; j < NTL; j++) {
                                const uint8_t *const xj = xb + j * 8u * act_stride(a.cols) + 64u * p;
                                const uint2 p0 = *reinterpret_cast<const uint2 *>(xj), p1 = *reinterpret_cast<const uint2 *>(xj + 32u);
                                const float2 dv0 = *reinterpret_cast<const float2 *>(sb0 + j * 8u * scale_stride(a.cols) + 8u * p);
                                const float2 dv1 = *reinterpret_cast<const float2 *>(sb1 + j * 8u * scale_stride(a.cols) + 8u * p);
                                int c0[4], c1[4];
                                mma_s8(c0, a00, a01, a02, a03, p0.x, p0.y);
                                mma_s8(c1, e00, e01, e02, e03, p1.x, p1.y);
#pragma unroll
                                for (int o = 0; o < 4; o++) {
                                    const float2 dv = (o & 1) ? dv1 : dv0;
                                    // (float with its offset) x sub-scale - offset x sub-scale: below 2^24, exact
                                    const float f0 = __fmaf_rn(__int_as_float(c0[o]), o < 2 ? l00 : l10, o < 2 ? k00 : k10);
                                    const float f1 = __fmaf_rn(__int_as_float(c1[o]), o < 2 ? l01 : l11, o < 2 ? k01 : k11);
                                    // (a plain last product would be fused into the addition that follows)
                                    const float v = __fmul_rn(o < 2 ? d0 : d1, __fmaf_rn(f0, dv.x, __fmul_rn(f1, dv.y)));
                                    if (p == 0 || p == 2) hold[j][o] = v;
                                    else if (p == 1) bs[j][o] = hold[j][o] + v;
                                    else bs[j][o] = bs[j][o] + (hold[j][o] + v);
                                }
                            }
                        }
                        // (a power-of-two row leaves a warp at most two blocks: pairwise)
#pragma unroll
                        for (int j = 0; j < NTL; j++)
#pragma unroll
                            for (int o = 0; o < 4; o++) sum[j][o] = b == b_lo ? bs[j][o] : sum[j][o] + bs[j][o];
                    }
                    if (a.ks_log) {   // the warps of the unit meet (one unit a chunk and warp), one fragment after the other
                        const uint32_t bar_n = 32u << a.ks_log, w0 = slot * ((1u << a.ks_log) - 1u);
#pragma unroll
                        for (int j = 0; j < NTL; j++) {
                            if (ks) *reinterpret_cast<float4 *>(it.red[w0 + ks - 1u][lane]) =
                                make_float4(sum[j][0], sum[j][1], sum[j][2], sum[j][3]);
                            asm volatile("bar.sync %0, %1;" ::"r"(1u + slot), "r"(bar_n) : "memory");
                            if (ks == 0) {
                                auto part = [&](uint32_t i, int o) { return it.red[w0 + i - 1u][lane][o]; };
#pragma unroll
                                for (int o = 0; o < 4; o++) {
                                    if (BB == 0) {
                                        for (uint32_t i = 1; i < 1u << a.ks_log; i++) sum[j][o] += part(i, o);
                                    } else if (a.ks_log == 1u) {
                                        sum[j][o] += part(1, o);
                                    } else if (a.ks_log == 2u) {
                                        sum[j][o] = (sum[j][o] + part(1, o)) + (part(2, o) + part(3, o));
                                    } else {
                                        sum[j][o] = ((sum[j][o] + part(1, o)) + (part(2, o) + part(3, o))) +
                                                    ((part(4, o) + part(5, o)) + (part(6, o) + part(7, o)));
                                    }
                                }
                            }
                            asm volatile("bar.sync %0, %1;" ::"r"(1u + slot), "r"(bar_n) : "memory");
                        }
                        if (ks) break;
                    }
                    float *const o0 = out + ch * rows_per_chunk + u * 16u + g;
#pragma unroll
                    for (int j = 0; j < NTL; j++)
#pragma unroll
                        for (uint32_t i = 0; i < 2; i++) {
                            const uint32_t r = 8u * j + 2u * t + i;
                            if (r < nr) {
                                o0[(uint64_t)r * a.ld_dst] = sum[j][i];
                                o0[(uint64_t)r * a.ld_dst + 8u] = sum[j][2 + i];
                            }
                        }
                }
                release();
            }
        };
        if (BB != 0 && nr == 1u) few(std::integral_constant<uint32_t, 1>{});
        else if (BB != 0 && nr == 2u) few(std::integral_constant<uint32_t, 2>{});
        else if (nr <= 8u) many(std::integral_constant<int, 1>{});
        else many(std::integral_constant<int, 2>{});
    });
}

// ---- host side ----
static bool g_ready = false;
constexpr uint32_t SMEM_MAX = 227u * 1024u;
template <uint32_t BB, uint32_t TPW> static bool warm_one() {
    return cudaFuncSetAttribute(wide_rows_k<BB, TPW>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX) == cudaSuccess;
}
bool warm() {
    g_ready = warm_one<1, 4>() && warm_one<2, 4>() && warm_one<4, 4>() && warm_one<8, 4>() && warm_one<0, 4>() &&
              warm_one<1, 2>() && warm_one<2, 2>() && warm_one<4, 2>() && warm_one<8, 2>() && warm_one<0, 2>();
    if (!g_ready) cudaGetLastError();
    return g_ready;
}

// Chunk and ring of a call.  Chunks of 64 tiles pay the barriers once per four tiles of a warp; a call with little
// work per CTA takes 32, so that its shares differ by less and its pipeline fills sooner.  (Items of 32 rows, three or
// four fragments a warp, were slower than two passes of 16: they spill, and their rows leave room for 32 tiles a
// chunk only: 370 experts of 32 rows 425 us against 284.)
static bool plan(Args &a) {
    const uint32_t B = a.cols >> 8, n_tiles = (a.w_rows >> 3) * B;
    const uint64_t tiles = (uint64_t)(a.w_rows >> 3) * B * a.n_entries;
    const bool small = tiles / 64u < 20ull * (uint64_t)g_q4b.n_sm;
    for (uint32_t want = small ? 32u : 64u; want >= 8u; want /= 2u) {
        // whole units of 16 weight rows (2 B tiles), a power of two of them so that all 16 warps get a share
        uint32_t units = 1;
        while (2u * units * 2u * B <= want) units *= 2u;
        a.ct = units * 2u * B;
        a.ks_log = 0;
        while ((units << (a.ks_log + 1u)) <= NCW && (2u << a.ks_log) <= B && a.ks_log < 3u) a.ks_log++;
        a.chunk_bytes = a.ct * Q4B_WIDE_BYTES;
        a.n_stage = MAX_STAGE;
        while (a.n_stage >= 2u && smem_bytes(a.cols, a.chunk_bytes, a.n_stage) > SMEM_MAX) a.n_stage--;
        if (a.n_stage >= 2u || want < 4u * B) break;
    }
    a.cpe = (n_tiles + a.ct - 1u) / a.ct;
    a.last_bytes = (n_tiles - (a.cpe - 1u) * a.ct) * Q4B_WIDE_BYTES;
    return a.n_stage >= 2u;
}
bool shape_ok(const uint8_t *w, uint64_t stride, uint64_t w_rows, uint64_t w_cols, uint32_t n_entries) {
    if (!g_ready || w_cols == 0 || (w_cols % 256u) || w_cols > 16384u || (w_rows % 16u) || n_entries > MAX_ENTRIES ||
        (stride % Q4B_TILE_BYTES) || !q4b_wide_of(w))
        return false;
    Args a = {};
    a.cols = (uint32_t)w_cols, a.w_rows = (uint32_t)w_rows, a.n_entries = n_entries;
    return plan(a);
}
template <uint32_t BB> static void launch_b(const Args &a, size_t sm) {
    if (a.ct > 32u || BB == 0) q4b_launch(wide_rows_k<BB, 4>, g_q4b.n_sm, NT, sm, g_q4b.stream, a);
    else q4b_launch(wide_rows_k<BB, 2>, g_q4b.n_sm, NT, sm, g_q4b.stream, a);
}
// a.w and a.expert_stride as the caller has them (tiled bytes)
bool launch(Args a) {
    a.w = q4b_wide_of(a.w);
    if (!a.w || !plan(a)) return false;
    a.expert_stride = a.expert_stride / Q4B_TILE_BYTES * Q4B_WIDE_BYTES;
    const size_t sm = smem_bytes(a.cols, a.chunk_bytes, a.n_stage);
    switch (a.cols >> 8) {
    case 1: launch_b<1>(a, sm); break;
    case 2: launch_b<2>(a, sm); break;
    case 4: launch_b<4>(a, sm); break;
    case 8: launch_b<8>(a, sm); break;
    default: launch_b<0>(a, sm); break;
    }
    return true;
}

}  // namespace wide
