// The tensor-core grouped product on the wide form of an arena (q4b_tile.cuh): the arithmetic of mmq_tc_k
// (q4b_mmq_tc.cu: fp16 operands that carry the scales, two planes of the activations, fp32 accumulators in
// tensor memory, one multiply by the super-block's d on the CUDA cores), for the calls in which there are
// 20 rows or more per possible entry (WIDE_TC_ROWS in q4b_grouped.cu, with both sides' times).  mmq_tc_k stays for arenas without a wide copy and for engine byte order.
//
// What bounded mmq_tc_k was neither its MMAs nor its decode but latency: with two steps of weight fields in
// registers ahead, a step of 128 x 128 weights took 3200 cycles when they came from HBM (512 experts of 17
// rows: 740 us for gate/up), of which the decode issues 440; and every 16 steps a new CTA filled its pipeline
// again.  Here:
//   - the kernel is persistent; a CTA walks its work items (a pass of up to 128 rows of an expert x a group of
//     weight-row tiles) as one pipeline, their descriptors fetched in batches ahead
//   - weights come by 16-byte cp.async into a ring that is private to each warp: no block barrier and
//     no dependence on what the L1 cache keeps
//   - the decoded operand goes to tensor memory (tcgen05.st), not to shared memory: writing 32 KB a step
//     there and having the MMAs read it back takes 512 cycles of a step's shared-memory bandwidth, and a fence
//   - a thread takes word t of the four groups of a step of its row: one AND-XOR and one fused half2
//     multiply-add for two weights, the four sub-scales by the same trick.  The k order that results (the
//     16 chunks of 8 values of a step transposed as 4 x 4, a chunk as 0 2 4 6 1 3 5 7) is the order in which
//     planes_k<true> writes the activations
//   - a pass's N is its own row count rounded up to the copy box of 16, and an expert's rows are split
//     evenly over its passes
#include "q4b_tile.cuh"

#include <atomic>

extern std::atomic<uint64_t> g_q4b_launches;
const uint8_t *q4b_wide_of(const void *p);

namespace mmqtc {

constexpr uint32_t W_ITEMS = 128;      // work items whose descriptors a CTA holds at a time
constexpr uint32_t W_NB = 128;         // rows of a pass at most
constexpr uint32_t W_BOX = 16;         // rows per activation copy: a pass's N is a multiple of it
constexpr uint32_t W_STAGES = 3;       // activation stages
constexpr uint32_t W_DG = 1;           // super-blocks of weights in flight per warp, 1 KB each
constexpr uint32_t W_NSL = W_NB / 64;  // 16-column slabs of an accumulator per epilogue thread
constexpr uint32_t W_REC = 8;          // super-blocks of records in the ring
constexpr uint32_t W_NA = 4;           // weight operand buffers in tensor memory, 64 columns each
constexpr uint32_t W_LAG = 2;          // super-blocks by which the records run ahead of the words
constexpr uint32_t W_A_COL = 256;      // the accumulators take the columns below
struct WItem {
    uint64_t mat;                      // wide bytes from the first expert's matrix to this item's first weight row
    int32_t rc;                        // first activation row
    uint32_t nrows;                    // rows of the pass
    uint32_t row0;                     // first weight row
    uint32_t pad;
};
struct __align__(1024) WSmem {
    uint2 rec[W_REC][MT];              // records (d, sub-scales) of the rows
    uint16_t dr[8][MT];                // d of the last super-blocks, for the epilogue
    WItem items[W_ITEMS];
    unsigned long long bar_mma[W_NA], a_full[W_NA], acc_empty[4], bar_b[4], b_empty[4];
    uint32_t tmem_base, n_items;
};
constexpr uint32_t W_B_OFF = (uint32_t)((sizeof(WSmem) + 1023u) & ~1023u);   // then activation stages, weight ring

struct WArgs {
    const uint8_t *w;                  // wide form of expert 0's matrix
    uint64_t expert_stride;            // wide bytes
    const int32_t *act;
    uint32_t cols, w_rows;
    float *dst;
    uint64_t ld_dst;
    uint32_t *err;
    const uint4 *work;                 // (entry, first row, rows) per pass
    const uint32_t *n_work;
    uint32_t groups, mt;               // an item is one of `groups` runs of mt 128-row tiles
    const float *rs;
};
constexpr uint32_t W_STAGE_BYTES = 4u * W_NB * 128u;   // two planes of two atoms of 64 k
constexpr uint32_t W_SMEM = W_B_OFF + W_STAGES * W_STAGE_BYTES + W_DG * NDW * 1024u;
static_assert(W_SMEM <= 227u * 1024u, "shared memory layout");

// The passes of every entry: its rows split evenly over as few passes of nb rows as hold them.
__global__ void __launch_bounds__(1024) worklist_wide_k(const int32_t *bounds,
                                                        const uint32_t *n_act, uint32_t n_entries,
                                                        uint4 *__restrict__ work,
                                                        uint32_t *__restrict__ n_work, uint32_t cap) {
    __shared__ uint32_t wsum[32];
    q4b_pdl_wait();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t n_ent = n_act ? min(*n_act, n_entries) : n_entries;
    uint32_t base = 0;
    for (uint32_t e0 = 0; e0 < n_ent; e0 += blockDim.x) {
        const uint32_t e = e0 + tid;
        const int32_t r0 = e < n_ent ? bounds[e] : 0;
        const uint32_t nr = e < n_ent ? (uint32_t)max(bounds[e + 1] - r0, 0) : 0u;
        const uint32_t np = (nr + W_NB - 1u) / W_NB, per = np ? (nr + np - 1u) / np : 0u;
        uint32_t inc = np;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= (uint32_t)o) inc += t;
        }
        if (lane == 31u) wsum[warp] = inc;
        __syncthreads();
        uint32_t pos = base + inc - np, tot = 0;
        for (uint32_t wv = 0; wv < 32u; wv++) {
            if (wv < warp) pos += wsum[wv];
            tot += wsum[wv];
        }
        for (uint32_t p = 0; p < np; p++, pos++)
            if (pos < cap) work[pos] = make_uint4(e, (uint32_t)r0 + p * per, min(per, nr - p * per), 0u);
        base += tot;
        __syncthreads();
    }
    if (tid == 0) *n_work = min(base, cap);
}

// One look at a barrier.
__device__ __forceinline__ bool mbar_look(unsigned long long *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// One lane of a converged warp.  (Known to the compiler as uniform: with lane == 0 in its place every operand of a
// tcgen05 instruction goes through a per-thread register, and issuing the 8 MMAs of a step took 880 cycles.)
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t *v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
// D (+)= A * B with A (128 rows x 16 k, fp16) in tensor memory
__device__ __forceinline__ void mma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        :
        : "r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }
__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<const uint32_t *>(&v); }

// Eight weights of a group (one word of the wide form) times its sub-scale ls, as fp16 integers in the
// order 0 2 | 4 6 | 1 3 | 5 7.  A nibble c' shifted up by one and combined with the exponent of 1024 is
// 1024 + 16 + w (low nibbles) or 1024 + 256 + 16 w (high nibbles); the fused multiply-add takes the offset off:
// every operand and result is an integer (or a sixteenth of ls) that fp16 holds exactly.
__device__ __forceinline__ uint4 decode_word_h(uint32_t x, __half2 L, __half2 C, __half2 L16, __half2 C16) {
    const uint32_t t = x << 1, u = x >> 7;
    uint4 r;
    r.x = h2_bits(__hfma2(as_h2((t & 0x001e001eu) ^ 0x64116411u), L, C));
    r.y = h2_bits(__hfma2(as_h2((t & 0x01e001e0u) ^ 0x65106510u), L16, C16));
    r.z = h2_bits(__hfma2(as_h2((u & 0x001e001eu) ^ 0x64116411u), L, C));
    r.w = h2_bits(__hfma2(as_h2((u & 0x01e001e0u) ^ 0x65106510u), L16, C16));
    return r;
}

// store_tile (q4b_mmq_tc.cu) with the row scales held by the warp's lanes: column j's by lane at + j.  (Loaded there, they
// would have to be loaded before the first store, which could alias them.)
__device__ __noinline__ void store_tile_lanes(float *o, uint64_t ld, float rs, uint32_t at, uint32_t n, float4 a0, float4 a1,
                                              float4 a2, float4 a3) {
    const float v[16] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w, a2.x, a2.y, a2.z, a2.w, a3.x, a3.y, a3.z, a3.w};
#pragma unroll
    for (uint32_t j = 0; j < 16; j++) {
        const float s = __shfl_sync(0xffffffffu, rs, at + j);
        if (j < n) o[(uint64_t)j * ld] = v[j] * s;
    }
}

// An accumulator is one step (128 k): the MMAs of the second activation plane, whose products are 2^-11 of the others',
// go in before those of the first, so that it takes eight full-size additions (mmq_tc_k: sixteen, each plane in
// columns of its own) and the epilogue reads one number per element.  Two accumulators alternate.  An epilogue thread
// owns two slabs of 16 columns.
__global__ void __launch_bounds__(NT, 1) mmq_wide_k(const WArgs a, const __grid_constant__ CUtensorMap map_h1,
                                                    const __grid_constant__ CUtensorMap map_h2) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    WSmem &s = *reinterpret_cast<WSmem *>(smem_raw);
    uint8_t *const sb_base = smem_raw + W_B_OFF;
    constexpr uint32_t stage_bytes = W_STAGE_BYTES;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    q4b_pdl_wait();
    const uint32_t B = a.cols >> 8, n_it = a.cols / KS, n_s = n_it * a.mt;   // steps of a tile, of an item
    const uint32_t n_all = *a.n_work * a.groups;
    if (blockIdx.x >= n_all) return;
    const uint32_t n_mine = (n_all - blockIdx.x + gridDim.x - 1u) / gridDim.x;
    const uint32_t tmem_cols = 512;   // two accumulators, four operand buffers
    if (tid == 0) {
        for (uint32_t i = 0; i < W_NA; i++) mbar_init(&s.bar_mma[i], 1), mbar_init(&s.a_full[i], NDW);
        for (uint32_t i = 0; i < NACC; i++) mbar_init(&s.acc_empty[i], NDW);
        for (uint32_t i = 0; i < 4; i++) mbar_init(&s.bar_b[i], 1), mbar_init(&s.b_empty[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem_base)),
                     "r"(tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s.tmem_base;
    // Bounded: half a second, then the error word, and from there on short waits.  A waiting warp sleeps between looks:
    // polling took issue slots from the decode warps (512 experts of 128 rows, an earlier version under ncu: 508 -> 463 us).
    unsigned long long patience = 500000000ull;
    auto wait = [&](unsigned long long *bar, uint32_t parity, uint32_t code) {
        if (mbar_look(bar, parity)) return;
        unsigned long long t0, t;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
        for (;;) {
            __nanosleep(100);
            if (mbar_look(bar, parity)) return;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
            if (t - t0 > patience) break;
        }
        atomicOr(a.err, ERR_MMQ_TC | code);
        patience = 10000ull;
    };
    // step counters run on over the batches: barrier phases follow them
    uint32_t it = 0;        // steps issued (MMA, copies) or decoded before this batch
    for (uint32_t first = 0; first < n_mine; first += W_ITEMS) {
        const uint32_t n_here = min(n_mine - first, W_ITEMS);
        if (first) __syncthreads();            // everybody is through with the batch before
        if (tid < n_here) {
            const uint32_t id = blockIdx.x + (first + tid) * gridDim.x, pass = id / a.groups, gr = id - pass * a.groups;
            const uint4 w = a.work[pass];
            WItem &m = s.items[tid];
            m.row0 = gr * a.mt * MT;
            m.mat = (uint64_t)(a.act ? a.act[w.x] : (int32_t)w.x) * a.expert_stride;
            m.rc = (int32_t)w.y;
            m.nrows = w.z;
        }
        __syncthreads();
        if (warp == NDW) {
            // ---- the MMA warp (one lane) ----
            if (elect_one()) {
                const uint64_t b_d0 = smem_desc_sw128(smem_u32(sb_base));
                const uint32_t b_lo0 = (uint32_t)b_d0, b_hi = (uint32_t)(b_d0 >> 32);
                uint32_t sb = it % W_STAGES, sb_ph = (it / W_STAGES) & 1u, j = it, buf = it % W_NA, buf_ph = (it / W_NA) & 1u;
                for (uint32_t i = 0; i < n_here; i++) {
                    const uint32_t np = (s.items[i].nrows + W_BOX - 1u) / W_BOX * W_BOX;
                    const uint32_t idesc = instr_desc(np), plane = (np * 128u) >> 4;
                    for (uint32_t k = 0; k < n_s; k++, j++) {
                        if (j >= NACC) wait(&s.acc_empty[j % NACC], (j / NACC - 1u) & 1u, 4u);
                        wait(&s.bar_b[sb], sb_ph, 1u);
                        wait(&s.a_full[buf], buf_ph, 8u);
                        tc_fence_after();
                        const uint32_t b_lo = b_lo0 + sb * (stage_bytes >> 4), d_addr = tmem + (j % NACC) * W_NB;
                        const uint32_t a_addr = tmem + W_A_COL + buf * 64u;
#pragma unroll
                        for (uint32_t c = 0; c < 16; c++) {
                            const uint32_t k = c & 7u;
                            mma_f16_ta(d_addr, a_addr + 8u * k,
                                       desc64(b_lo + (k >> 2) * 2u * plane + (k & 3u) * 2u + (c < 8u ? plane : 0u), b_hi), idesc, c ? 1u : 0u);
                        }
                        mma_commit(&s.bar_mma[buf]);
                        mma_commit(&s.b_empty[sb]);
                        if (++sb == W_STAGES) sb = 0, sb_ph ^= 1u;
                        if (++buf == W_NA) buf = 0, buf_ph ^= 1u;
                    }
                }
            }
        } else if (warp == NDW + 1u) {
            // ---- the copy warp (one lane): both activation planes of a step ----
            if (elect_one()) {
                uint32_t sb = it % W_STAGES, ph = (it / W_STAGES) & 1u, j = it;
                for (uint32_t i = 0; i < n_here; i++) {
                    const uint32_t np = (s.items[i].nrows + W_BOX - 1u) / W_BOX * W_BOX;
                    const int rc = s.items[i].rc;
                    uint32_t kt = 0;    // step within the tile: every tile reads the same rows again
                    for (uint32_t k = 0; k < n_s; k++, j++) {
                        if (j >= W_STAGES) wait(&s.b_empty[sb], ph ^ 1u, 16u);
                        mbar_expect_tx(&s.bar_b[sb], 4u * np * 128u);
#pragma unroll
                        for (uint32_t at = 0; at < 2; at++) {
                            uint8_t *dst = sb_base + sb * stage_bytes + at * 2u * np * 128u;
                            for (uint32_t r = 0; r < np; r += W_BOX) {
                                tma_load_2d(dst + r * 128u, &map_h1, &s.bar_b[sb], (int)(kt * KS + at * 64u), rc + (int)r);
                                tma_load_2d(dst + (np + r) * 128u, &map_h2, &s.bar_b[sb], (int)(kt * KS + at * 64u), rc + (int)r);
                            }
                        }
                        if (++kt == n_it) kt = 0;
                        if (++sb == W_STAGES) sb = 0, ph ^= 1u;
                    }
                }
            }
        } else {
            // ---- the 16 decode + epilogue warps: a super-block (two steps) per turn ----
            // decode: warp (t, quadrant) takes word t of every group of 32 rows, a lane a row (= a lane of tensor memory);
            // its k of a step are columns 16 t .. 16 t + 15 of the operand buffer
            const uint32_t e_q = warp & 3u, d_t = warp >> 2, e_row = 32u * e_q + lane;
            const uint32_t lane_base = (32u * e_q) << 16;
            const uint32_t ring = smem_u32(sb_base + W_STAGES * stage_bytes) + warp * 1024u;
            constexpr uint32_t SLOT = NDW * 1024u, DG = W_DG;
            // a row's 32 bytes of a super-block lie in the ring at 32 row, halves swapped in every second four rows
            const uint32_t rd = ring + lane * 32u, rx = ((lane >> 2) & 1u) << 4;
            // a copy instruction brings 16 rows, two lanes a row; the second 16 rows follow 2 B tiles later
            const uint32_t l_row = lane >> 1, wr = ring + l_row * 32u + (((lane & 1u) ^ ((l_row >> 2) & 1u)) << 4);
            // epilogue: of the pass's columns the slabs e_cs and e_cs + 4
            const uint32_t e_cs = warp >> 2;
            const uint32_t e_taddr = tmem + lane_base + 16u * e_cs;
            float acc[W_NSL][16];
#pragma unroll
            for (uint32_t h = 0; h < W_NSL; h++)
#pragma unroll
                for (int c = 0; c < 16; c++) acc[h][c] = 0.f;
            const uint32_t g0 = it >> 1, g_end = (it + n_here * n_s) >> 1;   // super-blocks of this batch

            // -- where a stream over the super-blocks of the batch's items stands: (item, super-block of the item, of the
            // tile), block of the byte tile, that byte tile's part t for this lane's row.  After eight super-blocks a row
            // goes on in the next byte tile (or, for rows of 1, 2, 4 or 8 super-blocks, has ended before).
            struct Place {
                uint32_t i = 0, b = 0, tb = 0, blk = 0, row = 0;
                const uint8_t *p = nullptr;
            };
            auto seek = [&](Place &f, uint32_t row, uint32_t off) {   // at the start of a tile
                if (f.tb) return;
                if (f.b == 0) f.row = s.items[f.i].row0 + row;
                const uint32_t bi = f.row * B;
                f.blk = bi & 7u;
                f.p = a.w + s.items[f.i].mat + (uint64_t)(bi >> 3) * Q4B_WIDE_BYTES + off;
                f.row += MT;
            };
            auto advance = [&](Place &f) {
                if (++f.blk == 8u) f.blk = 0, f.p += Q4B_WIDE_BYTES;
                if (++f.tb == B) f.tb = 0;
                if (++f.b == n_s / 2u) f.b = 0, f.i++;
            };
            Place fw, fr;
            const uint32_t second = 2u * B * Q4B_WIDE_BYTES, rec0 = smem_u32(&s.rec[0][e_row]);
            auto fetch_rec = [&](uint32_t at) {    // the next super-block's records, by the warps t = 0
                if (d_t == 0 && fr.i < n_here) {
                    seek(fr, e_row, 256u);
                    cp_async8(rec0 + at * (MT * 8u), fr.p + Q4B_WIDE_PART * (fr.blk >> 1) + 8u * (fr.blk & 1u));
                    advance(fr);
                }
            };
            auto fetch = [&](uint32_t at) {        // the next super-block's words into ring slot `at`
                if (fw.i < n_here) {
                    seek(fw, 32u * e_q + l_row, Q4B_WIDE_PART * d_t + 16u * (lane & 1u));
                    cp_async16(wr + at * SLOT, fw.p + fw.blk * 32u);
                    cp_async16(wr + at * SLOT + 512u, fw.p + second + fw.blk * 32u);
                    advance(fw);
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            // -- the super-blocks to retire
            uint32_t r_i = 0, r_tb = 0, r_m = 0;
            uint32_t r_rows = s.items[0].nrows;
            static_assert(W_NSL == 2, "a lane holds the scale of one column of the two slabs");
            auto row_scale = [&](uint32_t i) {     // of this warp's columns of item i
                const uint32_t c = 16u * (e_cs + 4u * (lane >> 4)) + (lane & 15u);
                return c < s.items[i].nrows ? a.rs[s.items[i].rc + (int32_t)c] : 0.f;
            };
            float r_scale = row_scale(0);
            auto fold = [&](uint32_t g, uint32_t half) {    // fold a complete step's accumulator into the sums
                tc_fence_after();
                const float dr = __half2float(__ushort_as_half(s.dr[g & 7u][e_row]));
#pragma unroll
                for (uint32_t h = 0; h < W_NSL; h++) {
                    if (16u * (e_cs + 4u * h) < r_rows) {   // warp-uniform
                        uint32_t v[16];
                        tmem_ld16(e_taddr + half * W_NB + 64u * h, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int c = 0; c < 16; c++) acc[h][c] = fmaf(dr, __uint_as_float(v[c]), acc[h][c]);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&s.acc_empty[half]);
                if (half == 0) return;
                if (++r_tb == B) {   // the tile is complete: write its rows out
                    const WItem &m = s.items[r_i];
#pragma unroll
                    for (uint32_t h = 0; h < W_NSL; h++) {
                        const uint32_t cs = e_cs + 4u * h;
                        if (16u * cs < r_rows)
                            store_tile_lanes(a.dst + (uint64_t)(m.rc + 16 * (int32_t)cs) * a.ld_dst + m.row0 + r_m * MT + e_row,
                                             a.ld_dst, r_scale, 16u * h, min(16u, r_rows - 16u * cs),
                                             make_float4(acc[h][0], acc[h][1], acc[h][2], acc[h][3]),
                                             make_float4(acc[h][4], acc[h][5], acc[h][6], acc[h][7]),
                                             make_float4(acc[h][8], acc[h][9], acc[h][10], acc[h][11]),
                                             make_float4(acc[h][12], acc[h][13], acc[h][14], acc[h][15]));
#pragma unroll
                        for (int c = 0; c < 16; c++) acc[h][c] = 0.f;
                    }
                    r_tb = 0;
                    if (++r_m == a.mt) {
                        r_m = 0;
                        if (++r_i < n_here) r_rows = s.items[r_i].nrows, r_scale = row_scale(r_i);
                    }
                }
            };
            // Records run W_LAG super-blocks ahead of the words, in the same copy groups: the warps t = 0 know theirs of
            // super-block g to have landed when they decode g - W_LAG, and the others learn it from the completion of
            // that super-block's MMAs, which they wait for before they decode g (the first ones from a barrier).
            uint32_t at = g0 % DG, rec_at = g0 % W_REC;
            for (uint32_t u = 0; u < W_LAG; u++) fetch_rec((rec_at + u) % W_REC);
            asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
            for (uint32_t u = 0; u < DG; u++) {
                fetch_rec((rec_at + W_LAG + u) % W_REC);
                fetch((at + u) % DG);
            }
            cp_async_wait<DG>();
            asm volatile("bar.sync 1, %0;" ::"n"(32 * NDW) : "memory");
            uint32_t rec_next = (rec_at + W_LAG + DG) % W_REC;
            for (uint32_t g = g0; g < g_end; g++) {
                // its two operand buffers (those of g - 2, whose MMAs were waited for when they were folded), and the
                // phase of the ones before, which hold g - 1
                const uint32_t bsel = (g & 1u) * 2u, ph = ((g - 1u) >> 1) & 1u;
                const bool old = g > g0;
                cp_async_wait<DG - 1>();
                __syncwarp();
                uint4 xs[2];
#pragma unroll
                for (uint32_t h = 0; h < 2; h++)
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(xs[h].x), "=r"(xs[h].y), "=r"(xs[h].z), "=r"(xs[h].w)
                                 : "r"(rd + at * SLOT + ((h << 4) ^ rx))
                                 : "memory");
                const uint2 rec = s.rec[rec_at][e_row];
                if (d_t == 0) s.dr[g & 7u][e_row] = (uint16_t)rec.x;
                __syncwarp();
                fetch_rec(rec_next);
                fetch(at);             // into the slot just read
#pragma unroll
                for (uint32_t h = 0; h < 2; h++) {
                    const uint4 x = xs[h];
                    const uint32_t v = q4b_prmt(rec.y, rec.y, h ? 0x3232u : 0x1010u), v8 = v >> 8;
                    uint32_t r[16];
#pragma unroll
                    for (uint32_t j = 0; j < 4; j++) {
                        const uint32_t y = j < 2 ? v : v8;
                        const __half2 L = (j & 1u) ? __hfma2(as_h2((y & 0x00f000f0u) | 0x64006400u), __float2half2_rn(0.125f),
                                                             __float2half2_rn(-127.f))
                                                   : __hfma2(as_h2((y & 0x000f000fu) | 0x64006400u), __float2half2_rn(2.f),
                                                             __float2half2_rn(-2047.f));
                        const uint4 d = decode_word_h(j == 0 ? x.x : j == 1 ? x.y : j == 2 ? x.z : x.w, L,
                                                      __hmul2(L, __float2half2_rn(-1040.f)), __hmul2(L, __float2half2_rn(0.0625f)),
                                                      __hmul2(L, __float2half2_rn(-80.f)));
                        r[4 * j] = d.x, r[4 * j + 1] = d.y, r[4 * j + 2] = d.z, r[4 * j + 3] = d.w;
                    }
                    tc_fence_after();
                    tmem_st16(tmem + lane_base + W_A_COL + (bsel + h) * 64u + 16u * d_t, r);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&s.a_full[bsel + h]);
                    if (old) {       // the step two before: its sums are read while the MMAs of the last one run
                        wait(&s.bar_mma[(bsel ^ 2u) + h], ph, 2u);
                        fold(g - 1u, h);
                    }
                }
                if (++at == DG) at = 0;
                if (++rec_at == W_REC) rec_at = 0;
                if (++rec_next == W_REC) rec_next = 0;
            }
#pragma unroll
            for (uint32_t h = 0; h < 2; h++) {
                wait(&s.bar_mma[((g_end - 1u) & 1u) * 2u + h], ((g_end - 1u) >> 1) & 1u, 2u);
                fold(g_end - 1u, h);
            }
        }
        it += n_here * n_s;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
    }
}

// ---- host side ----
static uint4 *g_wwork = nullptr;       // two lists, used in turn (gate/up, then down)
static uint32_t *g_wn_work = nullptr;
static uint32_t g_wturn = 0;
static bool g_wide_ready = false;
bool warm_wide() {
    if (g_wide_ready) return true;
    if (!g_ready ||
        cudaFuncSetAttribute(mmq_wide_k, cudaFuncAttributeMaxDynamicSharedMemorySize, W_SMEM) != cudaSuccess ||
        cudaMalloc(&g_wwork, 2 * WORK_CAP * sizeof(uint4)) != cudaSuccess ||
        cudaMalloc(&g_wn_work, 2 * sizeof(uint32_t)) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return g_wide_ready = true;
}
bool wide_ok(const uint8_t *w, uint64_t stride, uint64_t rows, uint64_t w_rows, uint64_t w_cols, uint32_t n_entries) {
    return g_wide_ready && shape_ok(w_rows, w_cols) && (stride % Q4B_TILE_BYTES) == 0 && rows < 0x7fffffffull &&
           (uint64_t)n_entries + rows / W_NB <= WORK_CAP && q4b_wide_of(w);
}
// h1, h2, rs: the rows' planes, as planes_k<true> writes them.
bool launch_wide(const uint8_t *w, uint64_t expert_stride, const int32_t *act, const uint32_t *n_act, uint32_t n_entries,
                 const int32_t *bounds, const __half *h1, const __half *h2, const float *rs, uint64_t rows, uint32_t cols,
                 uint32_t w_rows, float *dst, uint64_t ld_dst) {
    WArgs a = {};
    a.w = q4b_wide_of(w);
    if (!a.w) return false;
    a.expert_stride = expert_stride / Q4B_TILE_BYTES * Q4B_WIDE_BYTES;
    a.act = act;
    a.cols = cols;
    a.w_rows = w_rows;
    a.dst = dst;
    a.ld_dst = ld_dst;
    a.err = g_q4b.err_d;
    a.rs = rs;
    CUtensorMap maps[2];
    for (int pl = 0; pl < 2; pl++) {
        const cuuint64_t dims[2] = {cols, rows};
        const cuuint64_t strides[1] = {(cuuint64_t)cols * 2u};
        const cuuint32_t box[2] = {64, W_BOX};
        const cuuint32_t es[2] = {1, 1};
        if (g_encode(&maps[pl], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void *)(pl ? h2 : h1), dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    const uint32_t turn = g_wturn++ & 1u;
    q4b_launch(worklist_wide_k, 1, 1024, 0, g_q4b.stream, bounds, n_act, n_entries, g_wwork + turn * WORK_CAP, g_wn_work + turn,
               WORK_CAP);
    a.work = g_wwork + turn * WORK_CAP;
    a.n_work = g_wn_work + turn;
    // about 16 steps an item, as many tiles as that takes
    const uint32_t n_tiles = w_rows / MT, n_it = cols / KS;
    a.mt = 1;
    for (uint32_t c = 1; c <= n_tiles && c * n_it <= 16u; c++)
        if (n_tiles % c == 0) a.mt = c;
    a.groups = n_tiles / a.mt;
    q4b_launch(mmq_wide_k, g_q4b.n_sm, NT, W_SMEM, g_q4b.stream, a, maps[0], maps[1]);
    g_q4b_launches += 2;
    return q4b_launch_ok("mmq_wide");
}
// The planes of quantised rows.
bool launch_planes_wide(const int8_t *q, const float *dq, __half *h1, __half *h2, float *rs, uint64_t rows, uint32_t cols) {
    const uint32_t tpr = cols / 8u < 256u ? cols / 8u : 256u, rpb = 256u / tpr;
    planes_k<true><<<(unsigned)((rows + rpb - 1) / rpb), 256, 0, g_q4b.stream>>>(q, dq, rows, cols, tpr, h1, h2, rs);
    g_q4b_launches++;
    return q4b_launch_ok("planes");
}

}  // namespace mmqtc
