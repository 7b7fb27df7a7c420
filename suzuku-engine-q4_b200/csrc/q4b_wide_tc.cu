// The tensor-core grouped product on the wide form of an arena (q4b_tile.cuh): the arithmetic of mmq_tc_k
// (q4b_mmq_tc.cu: fp16 operands that carry the scales, two planes of the activations, fp32 accumulators in
// tensor memory, one multiply by the super-block's d on the CUDA cores), for the calls in which there are
// 20 rows or more per possible entry (WIDE_TC_ROWS in q4b_grouped.cu, with both sides' times).  mmq_tc_k stays for arenas
// without a wide copy and for engine byte order.
//
// What bounded mmq_tc_k was neither its MMAs nor its decode but latency, and every 16 steps (a step: 128 k) a new CTA
// filled its pipeline again.  Here:
//   - the kernel is persistent; a pair of CTAs (a cluster, two SMs) walks its work items (a pass of up to 128 rows of an
//     expert x a group of weight-row tiles) as one pipeline, their descriptors fetched in batches ahead
//   - the pair multiplies as one (cta_group::2): each CTA decodes 128 weight rows of its own and brings half of the
//     pass's activations, which halves what a step reads of them from the L2 (64 KB a step and SM before, with 128 rows)
//   - a pass of more than 64 rows is multiplied in two parts, so that four accumulators of 64 columns are in flight with any
//     number of rows and a decoded operand serves both
//   - the warps have one task each: 8 decode, two sets of 4 add finished steps to their sums in registers, two issue the
//     MMAs (every second step a warp: an MMA costs its thread some 25 cycles, a look at a barrier 60 to 100), one issues the
//     copies.  They meet through mbarriers only.  Nothing between the CTAs is ordered by a release or acquire at cluster
//     scope (those wait for the thread's stores to global memory: 1780 cycles a step instead of 1020 in an earlier version):
//     what crosses is a tensor-memory read or a decoded operand, which the tcgen05 fences order
//   - weights come by 16-byte cp.async into a ring that is private to each warp, two super-blocks a row at a time; the
//     next item's are brought to the L2 meanwhile
//   - the decoded operand goes to tensor memory (tcgen05.st), not to shared memory: writing 32 KB a step
//     there and having the MMAs read it back takes 512 cycles of a step's shared-memory bandwidth, and a fence
//   - a thread takes words 2 h, 2 h + 1 of the four groups of a step of its row: one AND-XOR and one fused half2
//     multiply-add for two weights, the four sub-scales by the same trick.  The k order that results (the
//     16 chunks of 8 values of a step transposed as 4 x 4, a chunk as 0 2 4 6 1 3 5 7) is the order in which
//     planes_k<true> writes the activations
//   - a step's activations are one copy: a box of [plane][64 k][rows], a tensor map for each number of rows
//   - a part's N is its own row count rounded up to 32
//
// Measured (512 experts, gate/up 1024 x 2048 / down 2048 x 512, us of the kernel under the profiler), before (one CTA, 16
// warps that decode and then add, passes of 128 rows) and now: 32 rows an expert 345 / 203 -> 236 / 136, 64 rows 376 / 224 ->
// 283 / 157, 96 rows 454 / 273 -> 414 / 250, 176 rows 896 / 524 -> 745 / 415.  What bounds it: the issue slots that decode
// and sums share.  A step of 32 rows takes some 850 cycles, in which a version with fewer warps issued 529 instructions a
// scheduler (65 % of the slots; ALU pipe 60 %, tensor pipe 31 %).  Tried and slower, with 32 / 64 rows where this takes 236 /
// 283: 16 decode warps 264 / 311 (the adding warps no longer get their slots), two decode sets that take super-blocks in turn
// 245 / 295, accumulators of 128 columns 319 / 375, one lane of a warp per barrier 274, tighter polling 243 / 298.  One
// set of adding warps and passes of 64 rows is faster with few rows (226 / 274) and slower with 96 (530).
#include "q4b_tile.cuh"

#include <atomic>

extern std::atomic<uint64_t> g_q4b_launches;
const uint8_t *q4b_wide_of(const void *p);

namespace mmqtc {

constexpr uint32_t W_ITEMS = 128;      // work items whose descriptors a CTA holds at a time
constexpr uint32_t W_BOX = 32;         // a part's N is a multiple of it (A in tensor memory, two CTAs)
constexpr uint32_t W_NB = 128;         // rows of a pass at most
constexpr uint32_t W_HB = 64;          // rows that are multiplied at a time: a pass has one part or two
constexpr uint32_t W_ND = 8;           // decode warps
constexpr uint32_t W_NE = 8;           // epilogue warps: two sets
constexpr uint32_t W_NT = 32 * (W_ND + W_NE + 4);   // and a warpgroup: two that issue MMAs, one that copies
constexpr uint32_t W_DG = 2;           // pairs of super-blocks of weights in flight per decode warp
constexpr uint32_t W_SLOT = 4096 + 512;   // their words and records
constexpr uint32_t W_A_COL = 256;      // weight operand buffers, 128 columns a super-block; the accumulators take the columns below
constexpr uint32_t W_NACC = W_A_COL / W_HB;   // accumulators, two to an issuing warp
static_assert(W_NACC == 4, "accumulators");
constexpr uint32_t W_STAGE = W_HB / 2u * 512u;   // a CTA's half of a part's activations of a step: two planes of 128 k
constexpr uint32_t W_NSB = 8;          // stages
struct WItem {
    uint64_t mat;                      // wide bytes from the first expert's matrix to this item's first weight row
    int32_t rc;                        // first activation row
    uint32_t nrows;                    // rows of the pass
    uint32_t row0;                     // first weight row
};
struct __align__(1024) WSmem {
    uint16_t dr[8][MT];                // d of the last super-blocks, for the epilogue
    WItem items[W_ITEMS];
    // a super-block decoded, a step of it multiplied; a part's MMAs complete (for the copies, and for the epilogue set that takes
    // it), its accumulator read, its activations landed.  A barrier is waited for by the parity of a phase, so none may be
    // two phases from the one that a waiter looks for (tests/test_wide_pipeline.py runs the roles under random schedules).  Hence sums
    // by set AND accumulator: the accumulator takes a part again only when the one before has been read, and its reader has
    // then seen its phase.  (Four to a set in turn: what orders the parts of a set was in part the other issuing warp's wait.)
    // And an accumulator is used by one issuing warp, two each: it has itself waited for the use before the last one to be read
    // and issued the last one, so it is that one's phase it finds open or complete.  (All four in turn by either warp: a wait for
    // a part that the other had still to issue was passed on an older phase, and sums not yet read were overwritten.)  The
    // issuing warps are three steps apart at most (a_full, a_free), seven parts: a stage's landing is never two phases behind.
    unsigned long long a_full[2], a_free[4], done[W_NSB], sums[2][W_NACC], acc_empty[W_NACC], b_full[W_NSB];
    uint32_t tmem_base;
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
    uint32_t groups, mt;               // an item is one of `groups` runs of mt pairs of 128-row tiles
    const float *rs;
};
constexpr uint32_t W_PIECE = MT * Q4B_WIDE_BYTES / 16u;   // weights of a step
constexpr uint32_t W_RING_OFF = W_B_OFF + W_NSB * W_STAGE;
constexpr uint32_t W_SMEM = W_RING_OFF + W_ND * W_DG * W_SLOT;
static_assert(W_SMEM <= 227u * 1024u, "shared memory layout");

// The passes of every entry: W_NB rows each, the rest in the last.
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
        const uint32_t np = (nr + W_NB - 1u) / W_NB;
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
            if (pos < cap) work[pos] = make_uint4(e, (uint32_t)r0 + p * W_NB, min(W_NB, nr - p * W_NB), 0u);
        base += tot;
        __syncthreads();
    }
    if (tid == 0) *n_work = min(base, cap);
}

__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, unsigned long long *bar, int c0, int c1, int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cta.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
        : "memory");
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
// The address of a shared variable of the cluster's first CTA, and an arrival there.
__device__ __forceinline__ uint32_t leader_addr(const void *p) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// ... that publishes no memory (an accumulator has been read): a release waits for the thread's stores to global memory
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t addr) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// Arrives at a barrier in both CTAs when the MMAs issued so far are complete.
__device__ __forceinline__ void mma_commit2(unsigned long long *bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"((uint16_t)3)
                 : "memory");
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
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t *v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]),
        "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]),
        "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
// D (+)= A * B over the two CTAs of a cluster, 128 rows x 16 k of A (fp16) in the tensor memory of each
__device__ __forceinline__ void mma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
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

// An accumulator is one step (128 k): the MMAs of the second activation plane, whose products are 2^-11 of the others',
// go in before those of the first, so that it takes eight full-size additions (mmq_tc_k: sixteen, each plane in
// columns of its own) and the epilogue reads one number per element.
struct WMaps {
    CUtensorMap m[2];                  // boxes of 16, 32 rows: a CTA's half of a pass
};
__cluster_dims__(2, 1, 1) __global__ void __launch_bounds__(W_NT, 1) mmq_wide_k(const WArgs a, const __grid_constant__ WMaps maps) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    WSmem &s = *reinterpret_cast<WSmem *>(smem_raw);
    uint8_t *const sb_base = smem_raw + W_B_OFF;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t rank = blockIdx.x & 1u, pair = blockIdx.x >> 1, n_pair = gridDim.x >> 1;
    q4b_pdl_wait();
    const uint32_t B = a.cols >> 8, n_it = a.cols / KS, n_s = n_it * a.mt;   // steps of a tile, of an item
    const uint32_t n_all = *a.n_work * a.groups;
    if (pair >= n_all) return;
    const uint32_t n_mine = (n_all - pair + n_pair - 1u) / n_pair;
    const uint32_t tmem_cols = 512;   // accumulators, operand buffers of two super-blocks
    if (tid == 0) {
        // (the first CTA's weights are full when the second one's step is there, too)
        for (uint32_t i = 0; i < 2u; i++) mbar_init(&s.a_full[i], W_ND + (rank ? 0u : 1u));
        for (uint32_t i = 0; i < 4u; i++) mbar_init(&s.a_free[i], 1);
        for (uint32_t i = 0; i < W_NSB; i++) mbar_init(&s.done[i], 1);
        for (uint32_t i = 0; i < W_NACC; i++) mbar_init(&s.acc_empty[i], W_NE), mbar_init(&s.sums[0][i], 1), mbar_init(&s.sums[1][i], 1);
        for (uint32_t i = 0; i < W_NSB; i++) mbar_init(&s.b_full[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem_base)),
                     "r"(tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem = s.tmem_base;
    // Bounded: half a second, then the error word, and from there on short waits.
    unsigned long long patience = 500000000ull;
    auto late = [&](uint32_t tries, unsigned long long &t0) {     // has a wait lasted too long?
        if ((tries & 255u) != 255u) return false;
        unsigned long long t;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        if (t0 == 0) t0 = t;
        return t - t0 > patience;
    };
    auto wait = [&](unsigned long long *bar, uint32_t parity, uint32_t code) {
        unsigned long long t0 = 0;
        for (uint32_t n = 0; !mbar_look(bar, parity); n++)
            if (late(n, t0)) {
                atomicOr(a.err, ERR_MMQ_TC | code);
                patience = 10000ull;
                return;
            }
    };
    // this CTA's tile at or behind a row (of an odd number of tiles the second CTA's last one is the first CTA's, and not stored)
    auto tile_row = [&](uint32_t row) { return row < a.w_rows ? row : row - MT; };
    // A role's part of every batch of items: body(steps before the batch, items).  The counters of steps, and those of parts
    // that roles keep, run on over the batches: barrier phases follow them.  (The threads of a warp may come to the barrier
    // one by one: of some only one lane works.)
    auto batches = [&](auto body) {
        uint32_t it = 0;
        for (uint32_t first = 0; first < n_mine; first += W_ITEMS) {
            const uint32_t n_here = min(n_mine - first, W_ITEMS);
            if (first) asm volatile("barrier.sync 0;" ::: "memory");        // everybody is through with the batch before
            if (tid < n_here) {
                const uint32_t id = pair + (first + tid) * n_pair, pass = id / a.groups, gr = id - pass * a.groups;
                const uint4 w = a.work[pass];
                WItem &m = s.items[tid];
                m.row0 = gr * a.mt * (2u * MT) + rank * MT;
                m.mat = (uint64_t)(a.act ? a.act[w.x] : (int32_t)w.x) * a.expert_stride;
                m.rc = (int32_t)w.y;
                m.nrows = w.z;
            }
            asm volatile("barrier.sync 0;" ::: "memory");
            body(it, n_here);
            it += n_here * n_s;
        }
    };
    // 96 registers a thread at launch (61,440 a CTA), shared out anew: 104, 112 and 40 make 60,416.  (More for the
    // last warpgroup's sake: with 32 its MMA warps spill, 260 us instead of 236.)
    if (warp >= W_ND + W_NE) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == W_ND + W_NE && rank) {
            // ---- the second CTA: tells the first one that a super-block's operands are there ----
            uint32_t u = 0;
            batches([&](uint32_t it, uint32_t n_here) {
                if (elect_one()) {
                    uint32_t j = it;
                    for (uint32_t i = 0; i < n_here; i++) {
                        const uint32_t parts = 2u * (s.items[i].nrows > W_HB ? 2u : 1u);
                        for (uint32_t k = 0; k < n_s; k += 2u, j += 2u) {
                            for (uint32_t p = 0; p < parts; p++, u++) wait(&s.b_full[u % W_NSB], (u / W_NSB) & 1u, 1u);
                            wait(&s.a_full[(j >> 1) & 1u], (j >> 2) & 1u, 1u);
                            tc_fence_after();
                            tc_fence_before();
                            mbar_arrive_cluster(leader_addr(&s.a_full[(j >> 1) & 1u]));
                        }
                    }
                }
            });
        } else if (warp < W_ND + W_NE + 2u && !rank) {
            // ---- the first CTA: the MMAs of both, every second step a warp (one lane) ----
            uint32_t u = 0, v = 0, tile = 0;     // parts, this warp's parts, tiles
            batches([&](uint32_t it, uint32_t n_here) {
                if (elect_one()) {
                    const uint64_t b_d0 = smem_desc_sw128(smem_u32(sb_base));
                    const uint32_t b_lo0 = (uint32_t)b_d0, b_hi = (uint32_t)(b_d0 >> 32);
                    uint32_t j = it + (warp & 1u);
                    for (uint32_t i = 0; i < n_here; i++) {
                        const uint32_t rows = s.items[i].nrows, parts = rows > W_HB ? 2u : 1u;
                        for (uint32_t m = 0; m < a.mt; m++, tile++) {
                            u += (warp & 1u) * parts;
                            for (uint32_t k = warp & 1u; k < n_it; k += 2u, j += 2u, u += parts) {
                                wait(&s.a_full[(j >> 1) & 1u], (j >> 2) & 1u, 1u);
                                for (uint32_t p = 0; p < parts; p++, u++, v++) {
                                    const uint32_t np = (min(rows - W_HB * p, W_HB) + W_BOX - 1u) / W_BOX * W_BOX;
                                    const uint32_t idesc = instr_desc(np) + ((MT >> 4) << 24), atom = (np * 64u) >> 4, sb = u % W_NSB;
                                    const uint32_t acc = 2u * (warp & 1u) + (v & 1u);
                                    if (v >= 2u) wait(&s.acc_empty[acc], (v / 2u - 1u) & 1u, 4u);
                                    wait(&s.b_full[sb], (u / W_NSB) & 1u, 1u);
                                    tc_fence_after();
                                    const uint32_t d_addr = tmem + acc * W_HB, a_addr = tmem + W_A_COL + (j & 3u) * 64u;
                                    const uint32_t b_lo = b_lo0 + sb * (W_STAGE >> 4);
#pragma unroll
                                    for (uint32_t c = 0; c < 16; c++) {    // the second plane's first
                                        const uint32_t kc = c & 7u;
                                        mma_f16_ta(d_addr, a_addr + 8u * kc,
                                                   desc64(b_lo + ((kc >> 2) + (c < 8u ? 2u : 0u)) * atom + (kc & 3u) * 2u, b_hi), idesc, c ? 1u : 0u);
                                    }
                                    mma_commit2(&s.done[sb]);
                                    mma_commit2(&s.sums[parts == 2u ? p : tile & 1u][acc]);
                                }
                                mma_commit2(&s.a_free[j & 3u]);
                            }
                            u -= (warp & 1u) * parts;
                        }
                    }
                }
            });
        } else if (warp == W_ND + W_NE + 2u) {
            // ---- the copy warp (one lane): this CTA's half of a part's rows of a step, [plane][64 k][row], in one copy ----
            uint32_t u = 0;
            batches([&](uint32_t it, uint32_t n_here) {
                if (elect_one())
                    for (uint32_t i = 0; i < n_here; i++) {
                        const uint32_t rows = s.items[i].nrows;
                        for (uint32_t m = 0; m < a.mt; m++) {      // every tile reads the same rows again
                            // the weights of the next item are brought to the L2 a piece a step
                            const uint8_t *pre = nullptr;
                            if (i + 1u < n_here) {
                                const WItem &nx = s.items[i + 1u];
                                pre = a.w + nx.mat + (uint64_t)(tile_row(nx.row0 + m * 2u * MT) * B >> 3) * Q4B_WIDE_BYTES;
                            }
                            for (uint32_t k = 0; k < n_it; k++) {
                                for (uint32_t r0 = 0; r0 < rows; r0 += W_HB, u++) {
                                    const uint32_t nb = (min(rows - r0, W_HB) + W_BOX - 1u) / W_BOX, sb = u % W_NSB;
                                    if (u >= W_NSB) wait(&s.done[sb], (u / W_NSB - 1u) & 1u, 16u);
                                    mbar_expect_tx(&s.b_full[sb], nb * (W_BOX / 2u * 512u));
                                    tma_load_4d(sb_base + sb * W_STAGE, &maps.m[nb - 1u], &s.b_full[sb], 0,
                                                s.items[i].rc + (int32_t)(r0 + rank * nb * (W_BOX / 2u)), (int)(2u * k), 0);
                                }
                                if (pre) {
                                    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(pre), "r"(W_PIECE) : "memory");
                                    pre += W_PIECE;
                                }
                            }
                        }
                    }
            });
        } else {
            batches([](uint32_t, uint32_t) {});
        }
    } else if (warp >= W_ND) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
        // ---- the epilogue warps: rows 32 q .. 32 q + 31 of the weights.  Of passes of two parts a set takes one, of passes of
        // one the sets take every second tile, so that one's stores are behind the other's sums ----
        const uint32_t q = warp & 3u, set = (warp >> 2) & 1u, e_row = 32u * q + lane;
        const uint32_t e_addr = tmem + ((32u * q) << 16);
        const uint32_t empty0 = leader_addr(&s.acc_empty[0]);
        uint32_t v = 0, tile = 0, seen = 0;       // parts of an issuing warp, tiles, parity of the phases seen of each accumulator's sums
        batches([&](uint32_t it, uint32_t n_here) {
            float sum[W_HB / 16u][16];
#pragma unroll
            for (uint32_t h = 0; h < W_HB / 16u; h++)
#pragma unroll
                for (int c = 0; c < 16; c++) sum[h][c] = 0.f;
            auto add = [&](uint32_t h, const uint32_t *v, float dr) {
#pragma unroll
                for (int c = 0; c < 16; c++) sum[h][c] = fmaf(dr, __uint_as_float(v[c]), sum[h][c]);
            };
            uint32_t j = it;
            for (uint32_t i = 0; i < n_here; i++) {
                const uint32_t rows = s.items[i].nrows, parts = rows > W_HB ? 2u : 1u, first = parts == 2u ? W_HB * set : 0u;
                const uint32_t n = min(rows - first, W_HB), row0 = s.items[i].row0;
                const int32_t rc = s.items[i].rc + (int32_t)first;
                // a lane holds the scale of two columns
                const float sc0 = lane < n ? a.rs[rc + (int32_t)lane] : 0.f;
                const float sc1 = lane + 32u < n ? a.rs[rc + 32 + (int32_t)lane] : 0.f;
                for (uint32_t m = 0; m < a.mt; m++, tile++) {
                    const uint32_t v0 = v + (parts == 2u ? set : 0u);
                    v += n_it / 2u * parts;                  // (n_it is even: as many of either warp)
                    if (parts == 1u && (tile & 1u) != set) {
                        j += n_it;
                        continue;
                    }
                    for (uint32_t k = 0; k < n_it; k++, j++) {
                        const uint32_t acc = 2u * (k & 1u) + ((v0 + (k >> 1) * parts) & 1u);
                        wait(&s.sums[set][acc], (seen >> acc) & 1u, 32u);
                        seen ^= 1u << acc;
                        tc_fence_after();
                        const float dr = __half2float(__ushort_as_half(s.dr[(j >> 1) & 7u][e_row]));
                        const uint32_t at = e_addr + acc * W_HB, empty = empty0 + 8u * acc;
                        uint32_t v[2][16];
                        tmem_ld16(at, v[0]), tmem_ld16(at + 16u, v[1]);
                        tmem_ld_wait();
                        if (n > 32u) {
                            add(0, v[0], dr), add(1, v[1], dr);
                            tmem_ld16(at + 32u, v[0]), tmem_ld16(at + 48u, v[1]);
                            tmem_ld_wait();
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_cluster_relaxed(empty);      // the sums are in registers
                            add(2, v[0], dr), add(3, v[1], dr);
                        } else {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive_cluster_relaxed(empty);
                            add(0, v[0], dr), add(1, v[1], dr);
                        }
                    }
                    // the tile is complete: write its rows out
                    const uint32_t t_row = row0 + m * 2u * MT;
                    float *o = a.dst + (int64_t)rc * (int64_t)a.ld_dst + t_row + e_row;
                    const uint32_t n_out = t_row < a.w_rows ? n : 0u;
#pragma unroll
                    for (uint32_t c = 0; c < W_HB; c++) {
                        const float f = __shfl_sync(0xffffffffu, c < 32u ? sc0 : sc1, c & 31u);
                        if (c < n_out) *o = sum[c >> 4][c & 15u] * f;
                        o += a.ld_dst;
                        sum[c >> 4][c & 15u] = 0.f;
                    }
                }
            }
        });
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
        // ---- the decode warps: two super-blocks (four steps) per turn ----
        // warp (h, quadrant) takes words 2 h, 2 h + 1 of every group of 32 rows, a lane a row (= a lane of tensor memory);
        // its k of a step are columns 32 h .. 32 h + 31 of that step's half of the operand buffer
        const uint32_t q = warp & 3u, d_h = warp >> 2;
        const uint32_t a_addr = tmem + ((32u * q) << 16) + W_A_COL + 32u * d_h;
        const uint32_t ring = smem_u32(smem_raw + W_RING_OFF) + warp * (W_DG * W_SLOT);
        // Of a pair of super-blocks a slot holds [word][row][4 x 16 bytes], the 16-byte chunk c (super-block c / 2, step c % 2
        // of it) at place c ^ (row / 2 % 4), and [row][super-block] the records.  A copy instruction brings eight rows of
        // a word, four lanes a row: a row's 64 bytes are two or three sectors of 32.
        const uint32_t rd = ring + lane * 64u, rx = (lane >> 1) & 3u;
        const uint32_t l_row = lane >> 2, l_c = lane & 3u, l_sb = l_c >> 1;
        const uint32_t wr = ring + l_row * 64u + ((l_c ^ ((l_row >> 1) & 3u)) << 4);
        // records: lane (row, c) those of super-block c / 2 of rows row + 8 (c % 2) and 16 behind it
        const uint32_t wr_rec = ring + 4096u + (l_row + 8u * (l_c & 1u)) * 16u + l_sb * 8u;
        const uint32_t eight = B * Q4B_WIDE_BYTES;       // eight rows further
        batches([&](uint32_t it, uint32_t n_here) {
            // where the lane's stream over super-blocks of the batch's items stands: item, tile, super-block of the tile
            uint32_t f_i = 0, f_m = 0, f_tb = l_sb;
            auto fetch = [&](uint32_t slot) {        // the next pair's words and records
                while (f_tb >= B) {
                    f_tb -= B;
                    if (++f_m == a.mt) f_m = 0, f_i++;
                }
                if (f_i < n_here) {
                    const WItem &m = s.items[f_i];
                    const uint32_t bi = (tile_row(m.row0 + f_m * 2u * MT) + 32u * q + l_row) * B + f_tb, blk = bi & 7u;
                    const uint8_t *const tile = a.w + m.mat + (uint64_t)(bi >> 3) * Q4B_WIDE_BYTES;
                    const uint8_t *const src = tile + Q4B_WIDE_PART * 2u * d_h + 32u * blk + 16u * (l_c & 1u);
                    const uint32_t to = wr + slot * W_SLOT;
#pragma unroll
                    for (uint32_t r = 0; r < 4; r++) {
                        cp_async16(to + 512u * r, src + r * eight);
                        cp_async16(to + 2048u + 512u * r, src + Q4B_WIDE_PART + r * eight);
                    }
                    const uint8_t *const rec = tile + (l_c & 1u) * eight + Q4B_WIDE_PART * (blk >> 1) + 256u + 8u * (blk & 1u);
                    cp_async8(wr_rec + slot * W_SLOT, rec);
                    cp_async8(wr_rec + slot * W_SLOT + 256u, rec + 2u * eight);
                }
                f_tb += 2u;
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
#pragma unroll
            for (uint32_t u = 0; u < W_DG; u++) fetch(u);
            uint32_t slot = 0, g = it >> 1;
            const uint32_t g_end = (it + n_here * n_s) >> 1;
            while (g < g_end) {
                cp_async_wait<W_DG - 1>();
                __syncwarp();
#pragma unroll 1
                for (uint32_t u = 0; u < 2u && g < g_end; u++, g++) {
                    uint4 xs[2][2];
#pragma unroll
                    for (uint32_t h = 0; h < 2; h++)
#pragma unroll
                        for (uint32_t w = 0; w < 2; w++)
                            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                         : "=r"(xs[h][w].x), "=r"(xs[h][w].y), "=r"(xs[h][w].z), "=r"(xs[h][w].w)
                                         : "r"(rd + slot * W_SLOT + 2048u * w + (((2u * u + h) ^ rx) << 4))
                                         : "memory");
                    uint2 rec;
                    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];"
                                 : "=r"(rec.x), "=r"(rec.y)
                                 : "r"(ring + slot * W_SLOT + 4096u + lane * 16u + 8u * u)
                                 : "memory");
                    if (d_h == 0) s.dr[g & 7u][32u * q + lane] = (uint16_t)rec.x;
                    if (u == 1u || g + 1u == g_end) {
                        __syncwarp();
                        fetch(slot);             // into the slot just read
                    }
#pragma unroll
                    for (uint32_t h = 0; h < 2; h++) {
                        const uint32_t v = q4b_prmt(rec.y, rec.y, h ? 0x3232u : 0x1010u), v8 = v >> 8;
                        uint32_t r[32];
#pragma unroll
                        for (uint32_t g4 = 0; g4 < 4; g4++) {
                            const uint32_t y = g4 < 2 ? v : v8;
                            const __half2 L = (g4 & 1u) ? __hfma2(as_h2((y & 0x00f000f0u) | 0x64006400u), __float2half2_rn(0.125f),
                                                                  __float2half2_rn(-127.f))
                                                        : __hfma2(as_h2((y & 0x000f000fu) | 0x64006400u), __float2half2_rn(2.f),
                                                                  __float2half2_rn(-2047.f));
                            const __half2 C = __hmul2(L, __float2half2_rn(-1040.f)), L16 = __hmul2(L, __float2half2_rn(0.0625f)),
                                          C16 = __hmul2(L, __float2half2_rn(-80.f));
#pragma unroll
                            for (uint32_t w = 0; w < 2; w++) {
                                const uint4 x = xs[h][w];
                                const uint4 d = decode_word_h(g4 == 0 ? x.x : g4 == 1 ? x.y : g4 == 2 ? x.z : x.w, L, C, L16, C16);
                                uint32_t *const to = r + 16u * w + 4u * g4;
                                to[0] = d.x, to[1] = d.y, to[2] = d.z, to[3] = d.w;
                            }
                        }
                        // that half of the super-block that had this buffer has been multiplied
                        if (g >= 2u) wait(&s.a_free[2u * (g & 1u) + h], (g / 2u - 1u) & 1u, 2u);
                        tc_fence_after();
                        tmem_st32(a_addr + (g & 1u) * 128u + h * 64u, r);
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&s.a_full[g & 1u]);
                }
                if (++slot == W_DG) slot = 0;
            }
        });
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();          // neither CTA's memory goes while the other's MMAs or arrivals may still reach it
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
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
    WMaps maps;
    for (uint32_t i = 0; i < 2u; i++) {
        const cuuint64_t dims[4] = {64, rows, cols / 64u, 2};
        const cuuint64_t strides[3] = {(cuuint64_t)cols * 2u, 128, (cuuint64_t)((const uint8_t *)h2 - (const uint8_t *)h1)};
        const cuuint32_t box[4] = {64, W_BOX / 2u * (i + 1u), 2, 2};
        const cuuint32_t es[4] = {1, 1, 1, 1};
        if (g_encode(&maps.m[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, (void *)h1, dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    const uint32_t turn = g_wturn++ & 1u;
    q4b_launch(worklist_wide_k, 1, 1024, 0, g_q4b.stream, bounds, n_act, n_entries, g_wwork + turn * WORK_CAP, g_wn_work + turn,
               WORK_CAP);
    a.work = g_wwork + turn * WORK_CAP;
    a.n_work = g_wn_work + turn;
    // about 16 steps an item, as many pairs of tiles as that takes
    const uint32_t n_pt = (w_rows / MT + 1u) / 2u, n_it = cols / KS;
    a.mt = 1;
    for (uint32_t c = 1; c <= n_pt && c * n_it <= 16u; c++)
        if (n_pt % c == 0) a.mt = c;
    a.groups = n_pt / a.mt;
    q4b_launch(mmq_wide_k, g_q4b.n_sm & ~1u, W_NT, W_SMEM, g_q4b.stream, a, maps);
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
