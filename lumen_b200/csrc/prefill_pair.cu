// Prefill grouped expert products on CTA pairs (tcgen05, cta_group::2), the form of a one-GPU call. Expert-parallel calls:
// prefill_tc.cu. The products are the reference's moe_grouped_gate_up_swiglu / moe_grouped_down kernels (cuda/shaders/moe_grouped.cu:1202-1760,
// :2183-2598).
//
// What bounds it: the tensor cores, if their operands arrive. One CTA alone reads 96 bytes a clock of operands from its
// shared memory for MMAs of 128 x 256 x 16, next to 32 + 32 written by its producers and its copies; 128 is all there
// is. A pair multiplies 256 x 256 x 16: each CTA holds 128 rows of the weights and half of the columns, which its partner
// reads as well, so that 64 bytes a clock are read. A tile has up to 512 columns (two
// accumulator sets of 256, all of TMEM), so each dequantised weight serves twice as many columns as in the one-CTA form.
//
// Weights are the M operand of both products, [128 rows per CTA, k], and the columns the N operand:
//   gate/up  a tile is 128 rows of I: 64 per CTA, as 64 gate and 64 up rows in groups of eight (eight gate rows, then
//            the same eight up rows). In the 16 x 256-bit shape of tcgen05.ld a thread then has gate and up of the same
//            two outputs, and SwiGLU needs no exchange
//   down     a tile is 256 rows of H: 128 per CTA
// N is 32..256 in steps of 32 per set, so ragged tiles cost what they hold. Results go through stmatrix (transposed) into one
// of two small buffers of the warp and leave from there: gate/up 32 bytes of a column at a time by the warp's stores, down 64 bytes of
// 32 columns as one tiled copy (by stores the waits for a free accumulator of 8192 tokens are 47 instead of 30 us; the
// 32-byte rows of gate/up lose with tiled copies, 27 and 33 us).
//
// One CTA pair per two SMs, persistent; tiles are claimed from a device-wide counter by the first CTA of the pair.
// Warps of a CTA: 0-7 epilogue (16 of them for gate/up when the weights come by TMA), then 16 weight producers (with
// TMA-fed weights a copy warp instead), two copy warps for the columns, every second unit each, one thread for the MMAs (idle in the
// second CTA), one thread for the tiles (idle in the second CTA).
//
// Operands come through two rings: weights in stages of 128 rows x 128 inputs, columns in units of up to 128 rows x 128
// inputs, of which a stage takes one per set. A pass multiplies one unit with its stage. What a pass costs the issuing thread
// besides its products (~450 cycles, in order) bounds narrow tiles, hence 128 inputs, ONE barrier to wait for (the unit's bytes and, in a stage's
// first pass, its weights) and ONE commit (unit free, and the stage with its last pass): with two barriers and two commits
// for every 64 inputs a tile of 60 columns took ~1200 cycles a pass (1000 tokens, 279 us a call).
// The columns of gate/up are gathered by the copies themselves (tile::gather4 on the token rows): the plane of the tokens
// stays in L2, where the gathered rows (268 MB at 8192 tokens of 2048, K = 8, 54 us to write) did not.
//
// Measured against the one-CTA kernels, gate/up + down in a short run: 4096 Zipf-loaded tokens (H = 2048, I = 768, E = 128, K = 8, Q4_0)
// 235 + 146 -> 200 + 115 us (1032 and 897 TFLOP/s, 0.64 and 0.56 of the measured burst peak), 8192 tokens 380 + 237 -> 321 + 184;
// narrow tiles: 300 tokens, a whole call 192 -> 148 us.
//
// Every wait is bounded; on expiry the kernel raises the status word, lets its copies and MMAs end, frees its TMEM and returns.
#include "tc_weights.cuh"

namespace lumen {

namespace pair {

using namespace tc;

constexpr int PROD_WARPS = 16;
constexpr int UNITS = 4;                                 // of the columns' ring
constexpr int STAGE_BYTES = 2 * SUB_BYTES;               // weights: 128 rows x 128 inputs, as two swizzle atoms of 64
// The two forms. Wide: tiles of up to 512 columns; two stages of weights, units of 128 rows (this CTA's half of a set of 256).
// Narrow: tiles of up to 128 columns; four stages, units of 64 rows. A stage comes back to its producers after ~1500
// cycles (dequantised, announced, multiplied, committed): with two stages that is what a narrow tile waits for, not the
// dequantisation (62 columns an expert: 1190 cycles a pass, 1000 without it).
template <bool NARROW>
struct Form {
    static constexpr int cols = NARROW ? 128 : 512, stages = NARROW ? 4 : 2;
    static constexpr int unit_rows = NARROW ? 64 : 128, atom_bytes = unit_rows * 128, unit_bytes = 2 * atom_bytes;
    static constexpr int ring_bytes = stages * STAGE_BYTES + UNITS * unit_bytes;  // 192 KB both
};
constexpr int SCHED_RING = 8;                            // tile descriptors in flight between the scheduler and the roles
constexpr int MAX_AHEAD = 4;                             // tiles that are claimed ahead of the MMAs at most
constexpr int TMEM_COLS = 512;

template <int MODE, bool ATMA, bool NARROW>
struct Roles {
    static constexpr int epi = (ATMA && MODE == 0) ? 16 : 8, prod = ATMA ? 0 : PROD_WARPS;
    static constexpr int copies = ATMA ? 3 : 2;  // a set's columns each, the weights
    static constexpr int prod0 = epi, copy0 = epi + prod, mma = copy0 + copies, sched = mma + 1, threads = (sched + 1) * 32;
    // arrivals for a stage's weights: half of the producer warps of both CTAs | the copies' expected bytes
    static constexpr int weight_arrivals = ATMA ? 1 : prod;
    // an output buffer: 32 columns of the warp's 16 (gate/up) or 32 (down) rows, in the 32- or 64-byte swizzle of the tiled
    // copy, with which the eight rows of an stmatrix hit eight different 16-byte bank groups
    static constexpr int row_bytes = (MODE == 0) ? 32 : 64, out_bytes = 32 * row_bytes;
    static constexpr size_t smem = 1024 + (size_t)Form<NARROW>::ring_bytes + (size_t)epi * 2 * out_bytes;
};

struct Args {
    CUtensorMap tmap_n;   // columns [rows, kdim] f16, box 64 x 32 (gathered: token rows, box 64 x 1)
    CUtensorMap tmap_w;   // the same, box 64 x 128
    CUtensorMap tmap_o;   // down: results [columns, H] f16, box 32 x 32
    CUtensorMap tmap_a;   // ATMA: the experts' f16 matrices (gate/up: in groups of eight gate and eight up rows)
    LayerDev L;
    const int4* tiles;    // {expert, first column, columns, m-tile}
    int32_t* n_tiles;     // [0..1] tiles of the gate/up and the down list, [2..3] the kernels' tile counters
    __half* out16;        // gate/up: S16 [C, I] in the order down reads it; down: D16 [C, H]
    const int32_t* gather;       // gate/up: token row of a compact column (null = the columns are rows of their own)
    int n_cols;                  // compact columns of the call
    const int32_t* out_row_map;  // down: output row of compact column c (null = c itself)
    int32_t* status;
    int32_t* status_host;
    uint64_t wait_limit_ns;
    int debug_extra_tx;   // test hook: the first stage's barrier expects this many bytes too many
    int kdim;             // H (gate/up) or I (down)
    int out_ld;           // I or H
};

// --- pair-wide forms of the building blocks ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
    return r;
}
// the address, in the pair's window, of the same shared-memory location of CTA `rank`
__device__ __forceinline__ uint32_t map_to(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void arrive_at(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void arrive_release_at(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ bool try_acquire(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// mbar_wait for what the other CTA writes with ordinary stores (tile descriptors)
__device__ __forceinline__ bool wait_acquire(uint32_t bar, uint32_t parity, const AbortCtl& ac) {
    if (try_acquire(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    for (uint32_t i = 0;; ++i) {
        if (try_acquire(bar, parity)) return true;
        if ((i & 63u) == 63u) {
            if (*ac.flag) return false;
            if (globaltimer_ns() - t0 > ac.limit_ns) {
                *ac.flag = 1u;
                return false;
            }
        }
    }
}
// whether the phase is over, without waiting for it
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void mbar_arrive_n(uint32_t bar, uint32_t n) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(n) : "memory");
}
__device__ __forceinline__ void pause_ns(uint64_t ns) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < ns) {
    }
}
__device__ __forceinline__ void pair_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// D[256, N] (+)= A[256, 16] B[N, 16]^T over the pair: each CTA holds 128 rows of A and N / 2 rows of B at these addresses
__device__ __forceinline__ void umma2(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}
// make_desc of an address given in 16-byte units
__device__ __forceinline__ uint64_t desc_of(uint32_t lo) {
    return (uint64_t)(lo | (1u << 16)) | ((uint64_t)((1u << 14) | (2u << 29) | 64u) << 32);
}
// one arrival at this barrier of both CTAs once the MMAs issued so far are done
__device__ __forceinline__ void umma2_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"((uint16_t)3)
                 : "memory");
}
__device__ __forceinline__ uint32_t idesc2(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((256u >> 4) << 24); }
// copies whose bytes count on a barrier of the pair's first CTA
__device__ __forceinline__ void tma_pair_2d(uint32_t dst, const CUtensorMap* m, int x, int y, uint32_t cluster_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(cluster_bar)
        : "memory");
}
__device__ __forceinline__ void tma_pair_5d(uint32_t dst, const CUtensorMap* m, int x, int c1, int c2, int c3, int c4, uint32_t cluster_bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], "
        "[%7];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(cluster_bar)
        : "memory");
}
// four rows of 64 inputs each, one after the other
__device__ __forceinline__ void tma_pair_gather4(uint32_t dst, const CUtensorMap* m, int x, const int4& r, uint32_t cluster_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes.cta_group::2 "
        "[%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(r.x), "r"(r.y), "r"(r.z), "r"(r.w), "r"(cluster_bar)
        : "memory");
}
// 16 TMEM lanes x 32 columns in the accumulator-fragment shape: v[4j..4j+1] row lane / 4, columns 8j + 2 (lane % 4) and the
// next, v[4j+2..4j+3] row lane / 4 + 8
__device__ __forceinline__ void tmem_ld_frag32(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
// (see tmem_ld_fence8)
__device__ __forceinline__ void tmem_ld_fence16(uint32_t (&r)[16]) {
    asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                      "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
}
// four 8 x 8 matrices of 16-bit elements, each stored transposed; lane l gives the address of row l % 8 of matrix l / 8
__device__ __forceinline__ void stmatrix4_t(uint32_t addr, const uint32_t (&v)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3])
                 : "memory");
}
__device__ __forceinline__ uint32_t pack_f16(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// --- dequantisation ---------------------------------------------------------------------------------------------------
// A producer warp owns 16 rows x 128 inputs of this CTA's operand in every second stage: eight warps fill a stage, the other
// eight the next one, so that each has the time of two passes for one wait, one fence and one arrival. It keeps this many of its
// tiles on the way in registers (9 or 17 KB an SM and stage):
constexpr int PREFETCH = 2;

// Where a lane's chunks go in the operand: 16 bytes of row m at (m / 8) 1024 + (m % 8) 128 + ((chunk ^ m % 8) 16).
// A quarter warp is two rows g of four chunks each. Down: rows in order, the two rows' m % 8 agree in bit 2, and the odd
// one takes the second block first. Gate/up: rows in the order in which down reads their outputs, their m % 8
// differ in bit 2, and both take the same block. Either way eight lanes hit eight different bank groups.
template <int MODE>
struct Place {
    uint32_t off[2];  // first / second pass, row g
    static constexpr uint32_t row8 = (MODE == 0) ? 4096 : 1024;  // row g + 8 from there
    bool swap;
    __device__ __forceinline__ Place(int rtl, int lane) {
        const int g = lane >> 2, t = lane & 3;
        int m;
        if (MODE == 0) {
            const int op = rtl >> 2, rt = rtl & 3, hi = rt & 1, mm = g & 3;
            const int slot = 4 * (mm & 1) + 2 * hi + (mm >> 1);
            m = 64 * (rt >> 1) + 16 * (g >> 2) + 8 * op + slot;
            swap = false;
        } else {
            m = 16 * rtl + g;
            swap = (g & 1) != 0;
        }
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int second = p ^ (swap ? 1 : 0);
            off[p] = (uint32_t)((m >> 3) * 1024 + (m & 7) * 128 + ((((second << 2) + t) ^ (m & 7)) << 4));
        }
    }
};

// half a tile (16 rows x 64 inputs): q words of blocks 2 sub, 2 sub + 1, the blocks' f16 scales of rows g and g + 8
template <int Q, int MODE>
__device__ __forceinline__ void dequant(const uint4& q0, const uint4& q1, uint32_t s_g, uint32_t s_g8, uint32_t a_base, const Place<MODE>& pl,
                                        const UnpackConst& k) {
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            // (gate/up never swaps: the selections below fold away)
            const bool second = (MODE == 0) ? (p == 1) : ((p == 1) != pl.swap);
            const uint32_t sc = prmt(r ? s_g8 : s_g, 0u, second ? 0x3232u : 0x1010u);
            uint32_t w0, w1 = 0u;
            if constexpr (Q == Q4_0) {
                w0 = second ? (r ? q0.w : q0.z) : (r ? q0.y : q0.x);
            } else {
                w0 = second ? (r ? q1.z : q1.x) : (r ? q0.z : q0.x);
                w1 = second ? (r ? q1.w : q1.y) : (r ? q0.w : q0.y);
            }
            store_weights<Q>(a_base + pl.off[p] + r * Place<MODE>::row8, w0, w1, sc, k);
        }
}

// columns of set h of a tile, rounded up to what an MMA of the pair takes
__device__ __forceinline__ int set_cols(int ncols, int h) { return (min(256, ncols - 256 * h) + 31) & ~31; }

template <int Q, int MODE, bool ATMA, bool NARROW>
__global__ void __launch_bounds__(Roles<MODE, ATMA, NARROW>::threads, 1)
grouped_gemm_pair_kernel(const __grid_constant__ Args a) {
    using R = Roles<MODE, ATMA, NARROW>;
    using F = Form<NARROW>;
    constexpr int STAGES = F::stages, UNIT_BYTES = F::unit_bytes;
    extern __shared__ uint8_t smem_raw[];
    // "first": used in the pair's first CTA only, which both CTAs' roles arrive at
    __shared__ uint64_t full_bar[UNITS];       // first: what a pass multiplies is there in both CTAs
    __shared__ uint64_t done_bar[UNITS];       // a pass is over
    __shared__ uint64_t acc_full_bar[2];       // an accumulator set is complete
    __shared__ uint64_t acc_empty_bar[2];      // first: it has been read in both CTAs
    __shared__ uint64_t sched_full_bar[SCHED_RING];
    __shared__ uint64_t sched_empty_bar[SCHED_RING];  // first
    __shared__ uint64_t go_bar[MAX_AHEAD];     // first: the next tile may be claimed
    __shared__ uint64_t drain_bar;             // give-up path: the MMAs issued are done
    __shared__ int4 sched_tile_s[SCHED_RING];
    __shared__ int4 rows_s[2][32];             // a tile's token rows in fours, by set
    __shared__ uint32_t tmem_base_s;
    __shared__ uint32_t abort_s;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cta_rank();
    const uint32_t stage0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const AbortCtl abort_flag{&abort_s, a.wait_limit_ns};

    if (tid == 0) {
        abort_s = 0u;
        for (int i = 0; i < UNITS; ++i) {
            mbar_init(smem_u32(&full_bar[i]), R::weight_arrivals + 1);  // and the columns' copies
            mbar_init(smem_u32(&done_bar[i]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&acc_full_bar[b]), 1);
            mbar_init(smem_u32(&acc_empty_bar[b]), 2 * R::epi);
        }
        for (int s = 0; s < SCHED_RING; ++s) {
            mbar_init(smem_u32(&sched_full_bar[s]), 1);
            mbar_init(smem_u32(&sched_empty_bar[s]), 2 * (R::epi + R::prod + R::copies) + 1);  // readers: epilogue, producers, copies of both; MMAs
        }
        for (int i = 0; i < MAX_AHEAD; ++i) mbar_init(smem_u32(&go_bar[i]), 1);
        mbar_init(smem_u32(&drain_bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == R::mma) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"((uint32_t)TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    pair_sync();  // both CTAs' barriers exist before either arrives at the other's
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;

    grid_dep_sync();
    const int ntiles = a.n_tiles[MODE];
    const int kgs = a.kdim >> 7;  // 128-input groups: stages of a tile
    auto pass_done = [&](uint32_t n) -> bool { return mbar_wait(smem_u32(&done_bar[n % UNITS]), (n / UNITS) & 1, abort_flag); };
    const int cl = blockIdx.x >> 1, ncl = gridDim.x >> 1;
    const uint32_t sched_empty_first = map_to(smem_u32(&sched_empty_bar[0]), 0);

    // The n-th tile of the pair (n counted by the caller): false when the list is exhausted or the kernel gives up.
    auto take_tile = [&](bool whole_warp, int& n, int4& tile) -> bool {
        const int slot = n % SCHED_RING;
        bool ok = wait_acquire(smem_u32(&sched_full_bar[slot]), (n / SCHED_RING) & 1, abort_flag);
        if (whole_warp) ok = __all_sync(0xffffffffu, ok);
        if (!ok) return false;
        tile = sched_tile_s[slot];
        if (whole_warp) __syncwarp();
        if (!whole_warp || lane == 0) arrive_at(sched_empty_first + slot * 8);
        ++n;
        return whole_warp ? __all_sync(0xffffffffu, tile.z >= 0) : tile.z >= 0;
    };
    // How many tiles are claimed ahead of the MMAs, and at which stage of a tile they allow the next claim. Long tiles:
    // one ahead, late in a wide tile so that the last tiles go to the pairs that are free first (before the producers need
    // it: they hold up to four groups and two stages beyond the MMAs), at the start of a narrow one, which
    // is over in about the time of a claim. Short ones: two ahead, so that the producers never run dry; four
    // where a tile is one group, because the producers' registers hold more than two of them.
    // (Narrow form: two more stages beyond the MMAs, passes of less than half the time.)
    const int ahead = NARROW ? (kgs >= 8 ? 2 : MAX_AHEAD) : (kgs >= 12) ? 1 : (kgs >= 2) ? 2 : MAX_AHEAD;

    if (warp < R::epi) {
        // ------------------------------ epilogue ------------------------------
        constexpr int PARTS = R::epi / 4;
        const int quad = warp & 3, part = warp >> 2;  // (TMEM lanes 32 quad.. are this warp's by the hardware's rule)
        const uint32_t buf0 = stage0 + F::ring_bytes + (uint32_t)warp * 2 * R::out_bytes;
        // 16-byte piece pc of row (column) cc of a buffer
        auto piece = [&](int cc, int pc) -> uint32_t {
            return (MODE == 0) ? cc * 32 + ((pc ^ ((cc >> 2) & 1)) << 4) : cc * 64 + ((pc ^ ((cc >> 1) & 3)) << 4);
        };
        int chunk = 0;  // this warp's so far: its parity is the buffer
        const uint32_t acc_empty_first = map_to(smem_u32(&acc_empty_bar[0]), 0);
        int v = 0, tn = 0;
        int4 tile;
        bool ok = true;
        while (ok && take_tile(true, tn, tile)) {
            const int nsets = (!NARROW && tile.z > 256) ? 2 : 1;
            // this warp's first output of a column's row
            const int o0 = (MODE == 0) ? tile.w * 128 + (int)rank * 64 + quad * 16 : tile.w * 256 + (int)rank * 128 + quad * 32;
            for (int h = 0; h < nsets; ++h, ++v) {
                const int set = v & 1;
                ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&acc_full_bar[set]), (v >> 1) & 1, abort_flag));
                if (!ok) break;
                tc_fence_after();
                const int ncols = min(256, tile.z - 256 * h), col0 = tile.y + 256 * h;
                const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + set * 256;
                // 32 columns of 16 rows into the buffer
                auto rows16 = [&](const uint32_t (&x)[16], int half, uint32_t buf) {
                    if (MODE == 0) {
                        uint32_t o[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            o[j] = pack_f16(swiglu_fast(__uint_as_float(x[4 * j]), __uint_as_float(x[4 * j + 2])),
                                            swiglu_fast(__uint_as_float(x[4 * j + 1]), __uint_as_float(x[4 * j + 3])));
                        stmatrix4_t(buf + piece(lane, half), o);
                    } else {
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            uint32_t o[4];
#pragma unroll
                            for (int j = 0; j < 4; ++j) o[j] = pack_f16(__uint_as_float(x[4 * j + 2 * q]), __uint_as_float(x[4 * j + 2 * q + 1]));
                            stmatrix4_t(buf + piece(lane, 2 * half + q), o);
                        }
                    }
                };
                // the TMEM loads of the next 16 rows are issued before the current ones are worked on
                uint32_t v0[16], v1[16];
                if (part * 32 < ncols) tmem_ld_frag32(taddr + part * 32, v0);
                for (int c = part * 32; c < ncols; c += PARTS * 32, ++chunk) {
                    const uint32_t buf = buf0 + (chunk & 1) * R::out_bytes;
                    tmem_ld_wait();
                    tmem_ld_fence16(v0);
                    tmem_ld_frag32(taddr + (16u << 16) + c, v1);
                    if (MODE == 1 && lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");  // the copy before the last has left its buffer
                    __syncwarp();
                    rows16(v0, 0, buf);
                    tmem_ld_wait();
                    tmem_ld_fence16(v1);
                    if (c + PARTS * 32 < ncols) tmem_ld_frag32(taddr + c + PARTS * 32, v0);
                    rows16(v1, 1, buf);
                    if (MODE == 1) fence_proxy_async();
                    __syncwarp();
                    const bool whole = MODE == 1 && c + 32 <= ncols && a.out_row_map == nullptr;
                    if (MODE == 1 && lane == 0) {
                        if (whole)
                            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                                             reinterpret_cast<uint64_t>(&a.tmap_o)),
                                         "r"(o0), "r"(col0 + c), "r"(buf)
                                         : "memory");
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");  // (one group a chunk, an empty one too)
                    }
                    if (!whole) {
                        constexpr int PIECES = R::row_bytes / 16;
#pragma unroll
                        for (int i = 0; i < PIECES; ++i) {
                            const int p = i * 32 + lane, cc = p / PIECES, pc = p % PIECES;
                            const uint4 x = lds128(buf + piece(cc, pc));
                            if (c + cc < ncols) {
                                int row = col0 + c + cc;
                                if (MODE == 1 && a.out_row_map != nullptr) row = a.out_row_map[row];
                                *reinterpret_cast<uint4*>(a.out16 + (size_t)row * a.out_ld + o0 + pc * 8) = x;
                            }
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) arrive_at(acc_empty_first + set * 8);
            }
        }
        if (MODE == 1 && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // every result has been written
        __syncwarp();
    } else if (warp < R::copy0) {
        // --------------------------- weight producers --------------------------
        if constexpr (!ATMA) {
            const int pw = warp - R::prod0, rtl = pw & 7;
            constexpr int NQ = QTraits<Q>::NQ;
            const Place<MODE> pl(rtl, lane);
            const UnpackConst k = unpack_const_pinned<Q>();
            const uint32_t full_first = map_to(smem_u32(&full_bar[0]), 0);
            // load cursor: this warp's next stage is group kg of the tile at hand, whose first pass is number u0
            int tn = 0, kg = (pw >> 3) - kgs;
            uint32_t u0 = 0;
            bool more = true;               // the list may hold further tiles
            int sets = 0, sets_before = 0;  // accumulator sets of the tile at hand and of the one before (0: none)
            const uint4 *qt = nullptr, *st = nullptr;
            WTile<Q> w[PREFETCH];
            uint32_t pass[PREFETCH];   // a slot's first pass
            uint32_t before[PREFETCH]; // the passes over which its stage is free
            bool there[PREFETCH];
            // the warp's next tile into registers; false when there is none. The descriptor of a tile that is still to be
            // claimed is waited for: it comes without any help from the tiles that are held here (see `ahead`)
            auto load_next = [&](int j) {
                kg += (sets == 0) ? kgs : 2;  // (the first call starts at the warp's own first group)
                while (sets == 0 || kg >= kgs) {
                    if (sets != 0) kg -= kgs;
                    int4 tile;
                    more = more && take_tile(true, tn, tile);
                    if (!more) {
                        there[j] = false;
                        return;
                    }
                    u0 += (uint32_t)(kgs * sets);
                    sets_before = sets;
                    sets = (!NARROW && tile.z > 256) ? 2 : 1;
                    const int e = tile.x;
                    const uint4 *qb, *sb;
                    int rt;
                    if (MODE == 0) {
                        const bool up = rtl >= 4;
                        qb = up ? a.L.up_q(e) : a.L.gate_q(e);
                        sb = up ? a.L.up_s(e) : a.L.gate_s(e);
                        rt = tile.w * 8 + (int)rank * 4 + (rtl & 3);
                    } else {
                        qb = a.L.down_q(e);
                        sb = a.L.down_s(e);
                        rt = tile.w * 16 + (int)rank * 8 + rtl;
                    }
                    const size_t tidx = (size_t)rt * kgs;
                    qt = qb + tidx * (NQ * 32) + lane;
                    st = sb + tidx * 8 + (lane >> 2);
                }
                const uint4* qp = qt + kg * (NQ * 32);
#pragma unroll
                for (int i = 0; i < NQ; ++i) w[j].q[i] = ldg_stream(qp + i * 32);
                w[j].s = ldg_stream(st + kg * 8);
                pass[j] = u0 + (uint32_t)(kg * sets);
                // stage n - 2 is over with the pass in front of stage n - 1's first
                if (!NARROW) before[j] = pass[j] - (uint32_t)(kg > 0 ? sets : sets_before);
                there[j] = true;
            };
#pragma unroll
            for (int j = 0; j < PREFETCH; ++j) load_next(j);
            uint32_t n = pw >> 3;  // stage
            bool ok = true;
            while (ok) {
#pragma unroll
                for (int j = 0; j < PREFETCH; ++j) {
                    ok = ok && there[j];
                    if (!ok) break;
                    if (n >= STAGES) ok = __all_sync(0xffffffffu, pass_done((NARROW ? n - STAGES + 1 : before[j]) - 1));
                    if (!ok) break;
                    const uint32_t base = stage0 + (n % STAGES) * STAGE_BYTES;
#pragma unroll
                    for (int sub = 0; sub < 2; ++sub)
                        dequant<Q, MODE>(w[j].q[Q == Q4_0 ? sub : (2 * sub) % NQ], w[j].q[Q == Q4_0 ? sub : (2 * sub + 1) % NQ], sub ? w[j].s.y : w[j].s.x,
                                         sub ? w[j].s.w : w[j].s.z, base + sub * SUB_BYTES, pl, k);
                    fence_proxy_async();  // every lane's own stores, before the warp's one arrival
                    __syncwarp();
                    if (lane == 0) arrive_at(full_first + ((NARROW ? n : pass[j]) % UNITS) * 8);
                    n += 2;
                    load_next(j);
                }
            }
        }
    } else if (warp < R::copy0 + 2) {
        // ------------------------- copies of the columns -----------------------
        // Each warp takes every second unit: one set of a wide tile's stages, every second stage of a narrow tile.
        const uint32_t w = warp - R::copy0;
        const uint32_t full_first = map_to(smem_u32(&full_bar[0]), 0);
        const uint32_t units0 = stage0 + STAGES * STAGE_BYTES;
        const bool gather = (MODE == 0) && a.gather != nullptr;
        int tn = 0;
        uint32_t u0 = 0;     // the tile's first unit
        uint32_t asked = 0;  // behind this warp's last unit on its way
        bool ok = true;
        // this CTA's rows of the warp's set of a tile that begins at unit u: `half` of them from the returned column on
        auto rows_of = [&](const int4& t, uint32_t u, int& half) -> int {
            const int h = (!NARROW && t.z > 256) ? (int)((w ^ u) & 1) : 0;
            half = set_cols(t.z, h) / 2;
            return t.y + 256 * h + (int)rank * half;
        };
        auto token_rows = [&](const int4& t, uint32_t u) -> int4 {
            int half;
            const int c = rows_of(t, u, half) + 4 * lane, last = a.n_cols - 1;
            if (4 * lane >= half) return make_int4(0, 0, 0, 0);
            return make_int4(__ldg(a.gather + min(c, last)), __ldg(a.gather + min(c + 1, last)), __ldg(a.gather + min(c + 2, last)),
                             __ldg(a.gather + min(c + 3, last)));
        };
        int4 tile, tile_n = make_int4(0, 0, -1, 0), rows_n = make_int4(0, 0, 0, 0);
        bool have = take_tile(true, tn, tile);
        if (have && gather) rows_n = token_rows(tile, 0);
        const int pre = max(kgs - 4, 0);  // where the next tile's descriptor and token rows are fetched
        while (ok && have) {
            const bool wide = !NARROW && tile.z > 256;
            int half;
            const int first = rows_of(tile, u0, half);
            const uint32_t bytes = 2 * (gather ? half * 128 : (half == 128) ? 128 * 128 : ((half + 31) / 32) * 4096);
            const uint32_t u_next = u0 + (wide ? 2 * kgs : kgs), odd = (w ^ u0) & 1;
            if (gather) {
                __syncwarp();
                rows_s[w][lane] = rows_n;
                __syncwarp();
            }
            bool fetched = false;
            auto fetch_next = [&]() {
                have = take_tile(true, tn, tile_n);
                if (have && gather) rows_n = token_rows(tile_n, u_next);
                fetched = true;
            };
            for (int k = wide ? 0 : (int)odd; k < kgs; k += wide ? 1 : 2) {
                if (k >= pre && !fetched) fetch_next();
                const uint32_t unit = u0 + (wide ? 2 * k + odd : k), s = unit % UNITS;
                ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&done_bar[s]), ((unit / UNITS) & 1) ^ 1, abort_flag));
                if (!ok) break;
                if (elect_one()) {
                    if (rank == 0) {
                        // both CTAs' bytes (their copies have the same shape) are expected once, by the first CTA; the second
                        // pass of a stage has no weights of its own to wait for
                        mbar_expect_tx(smem_u32(&full_bar[s]), 2 * bytes + (unit == 0 ? a.debug_extra_tx : 0));
                        if (wide && odd) mbar_arrive_n(smem_u32(&full_bar[s]), R::weight_arrivals);
                    }
                    const uint32_t dst = units0 + s * UNIT_BYTES, bar = full_first + s * 8;
                    const int x = k * 128;
                    if (gather) {
                        // (sixteen rows' numbers first: a load between two copies would cost its latency each time)
                        for (int q = 0; q < half / 4; q += 4) {
                            int4 r[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) r[i] = rows_s[w][q + i];
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                tma_pair_gather4(dst + (i & 1) * F::atom_bytes + (q + (i >> 1)) * 512, &a.tmap_n, x + (i & 1) * 64, r[i >> 1], bar);
                        }
                    } else if (!NARROW && half == 128) {
                        tma_pair_2d(dst, &a.tmap_w, x, first, bar);
                        tma_pair_2d(dst + F::atom_bytes, &a.tmap_w, x + 64, first, bar);
                    } else {
                        for (int q = 0; q * 32 < half; ++q) {
                            tma_pair_2d(dst + q * 4096, &a.tmap_n, x, first + q * 32, bar);
                            tma_pair_2d(dst + F::atom_bytes + q * 4096, &a.tmap_n, x + 64, first + q * 32, bar);
                        }
                    }
                }
                __syncwarp();
                asked = unit + 1;
            }
            if (!ok) break;
            if (!fetched) fetch_next();
            u0 = u_next;
            tile = tile_n;
        }
        // the copies land before the shared memory goes away (this warp's: every second unit up to the last one it asked for). The
        // second CTA cannot watch the first one's barriers: it waits longer than the first one does at most
        if (lane == 0 && *abort_flag.flag) {
            if (rank == 0) let_land(smem_u32(&full_bar[0]), UNITS, asked, 2);
            else pause_ns(UNITS * 1000000ull);
        }
        __syncwarp();
    } else if (ATMA && warp == R::copy0 + 2) {
        // ------------------------- copies of the weights -----------------------
        if (lane == 0) {
            const uint32_t full_first = map_to(smem_u32(&full_bar[0]), 0);
            int tn = 0;
            uint32_t n = 0, u = 0, last_1 = 0, last_2 = 0;  // as the producers count
            bool ok = true;
            int4 tile;
            while (ok && take_tile(false, tn, tile)) {
                for (int k = 0; k < kgs; ++k, ++n) {
                    ok = n < STAGES || pass_done(NARROW ? n - STAGES : last_2);
                    if (!ok) break;
                    const uint32_t s = u % UNITS, dst = stage0 + (n % STAGES) * STAGE_BYTES, bar = full_first + s * 8;
                    if (rank == 0) mbar_expect_tx(smem_u32(&full_bar[s]), 2 * STAGE_BYTES);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        if (MODE == 0)
                            tma_pair_5d(dst + i * SUB_BYTES, &a.tmap_a, k * 128 + i * 64, 0, 0, tile.w * 16 + (int)rank * 8, tile.x, bar);
                        else
                            tma_pair_2d(dst + i * SUB_BYTES, &a.tmap_a, k * 128 + i * 64, tile.x * a.L.H + tile.w * 256 + (int)rank * 128, bar);
                    }
                    u += (!NARROW && tile.z > 256) ? 2 : 1;
                    last_2 = last_1;
                    last_1 = u - 1;
                }
            }
            if (*abort_flag.flag) {
                if (rank == 0) let_land(smem_u32(&full_bar[0]), UNITS, u);
                else pause_ns(UNITS * 1000000ull);
            }
        }
        __syncwarp();
    } else if (warp == R::mma) {
        // -------------------------------- MMA ---------------------------------
        if (rank == 0 && elect_one()) {
            // (one thread in order: every instruction of a pass counts)
            const uint32_t a_base = (stage0 >> 4) & 0x3FFFu, b_base = ((stage0 + STAGES * STAGE_BYTES) >> 4) & 0x3FFFu;
            const uint32_t full0 = smem_u32(&full_bar[0]), done0 = smem_u32(&done_bar[0]);
            int tl = 0, tn = 0;
            uint32_t v = 0, u = 0, n = 0;  // accumulator sets, passes, stages so far
            bool ok = true, ready = false;  // ready: the next pass's operands are known to be there
            int4 tile;
            for (; ok && take_tile(false, tn, tile); ++tl) {
                const uint32_t wide = (!NARROW && (tile.z > 256)) ? 1u : 0u;
                const uint32_t id0 = idesc2(set_cols(tile.z, 0));
                const uint32_t id1 = idesc2(max(32, set_cols(tile.z, 1)));
                const uint32_t passes = (uint32_t)kgs << wide;
                const uint32_t go = (!NARROW && kgs >= 12 && (tile.z > 128)) ? (uint32_t)(kgs / 2 - 2) << wide : 0u;
                // The sets of a wide tile take turns, so that the first one is complete, and its epilogue under way, while the
                // second one's last products run, and the next tile's first products run under the second one's epilogue.
                for (uint32_t p = 0; p < passes; ++p, ++u) {
                    const uint32_t h = p & wide, set = (v + h) & 1, c = u % UNITS;
                    if (p == go) mbar_arrive(smem_u32(&go_bar[tl % ahead]));
                    if (p <= wide) ok = mbar_wait(smem_u32(&acc_empty_bar[set]), (((v + h) >> 1) & 1) ^ 1, abort_flag);
                    ok = (ok && (ready || mbar_wait(full0 + c * 8, (u / UNITS) & 1, abort_flag)));
                    if (!ok) break;
                    ready = mbar_test(full0 + ((u + 1) % UNITS) * 8, ((u + 1) / UNITS) & 1);  // (its answer comes under the products' issue)
                    tc_fence_after();
                    const uint32_t w_lo = a_base + (n % STAGES) * (STAGE_BYTES >> 4), c_lo = b_base + c * (UNIT_BYTES >> 4);
                    const uint32_t acc = tmem_base + set * 256, id = h ? id1 : id0;
                    {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const uint32_t ow = (j >> 2) * (SUB_BYTES >> 4) + (j & 3) * 2, oc = (j >> 2) * (F::atom_bytes >> 4) + (j & 3) * 2;
                            umma2(acc, desc_of(w_lo + ow), desc_of(c_lo + oc), id, (p > wide || j > 0) ? 1u : 0u);
                        }
                        umma2_commit(done0 + c * 8);
                        if (p + 1 + wide >= passes) umma2_commit(smem_u32(&acc_full_bar[set]));
                    }
                    n += (h == wide);
                }
                if (!ok) break;
                v += 1 + wide;
            }
            if (*abort_flag.flag) {
                // what has been issued reads both CTAs' shared memory: it ends before either goes away
                umma2_commit(smem_u32(&drain_bar));
                let_land(smem_u32(&drain_bar), 1, 1);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------ scheduler ------------------------------
        if (rank == 0 && lane == 0) {
            const uint32_t tile_other = map_to(smem_u32(&sched_tile_s[0]), 1), full_other = map_to(smem_u32(&sched_full_bar[0]), 1);
            for (int n = 0;; ++n) {
                const int slot = n % SCHED_RING, m = n - ahead;
                // tile n is claimed once the MMAs are far enough into tile n - ahead
                if (m >= 0 && !mbar_wait(smem_u32(&go_bar[m % ahead]), (m / ahead) & 1, abort_flag)) break;
                if (!wait_acquire(smem_u32(&sched_empty_bar[slot]), ((n / SCHED_RING) & 1) ^ 1, abort_flag)) break;
                // the first `ahead` tiles are the pair's by its index
                const int t = (n < ahead) ? cl + n * ncl : ahead * ncl + atomicAdd(a.n_tiles + 2 + MODE, 1);
                const int4 d = (t < ntiles) ? a.tiles[t] : make_int4(0, 0, -1, 0);  // columns < 0: no more tiles
                sched_tile_s[slot] = d;
                asm volatile("st.shared::cluster.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(tile_other + slot * 16), "r"(d.x), "r"(d.y), "r"(d.z), "r"(d.w)
                             : "memory");
                arrive_release_at(full_other + slot * 8);
                mbar_arrive(smem_u32(&sched_full_bar[slot]));
                if (t >= ntiles) break;
            }
        }
        __syncwarp();
    }

    tc_fence_before();
    __syncthreads();
    pair_sync();  // neither CTA leaves while the other may still arrive at its barriers or multiply from its shared memory
    if (warp == R::mma) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS) : "memory");
    }
    if (tid == 0 && abort_s) raise_status(a.status, a.status_host, 4);  // LUMEN_MOE_TIMEOUT
}

template <int Q, int MODE, bool ATMA, bool NARROW>
cudaError_t launch_one(const Args& a, int ctas, cudaStream_t st) {
    using R = Roles<MODE, ATMA, NARROW>;
    auto* kern = grouped_gemm_pair_kernel<Q, MODE, ATMA, NARROW>;
    static SmemOptIn optin;
    const cudaError_t e = ensure_dyn_smem(kern, R::smem, optin);
    if (e != cudaSuccess) return e;
    count_launch();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas & ~1);
    cfg.blockDim = dim3(R::threads);
    cfg.dynamicSmemBytes = R::smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kern, a);
}

template <int Q, bool ATMA, bool NARROW>
cudaError_t launch_both(const Args& gu, const Args& dn, int ctas, cudaStream_t st) {
    const cudaError_t e = launch_one<Q, 0, ATMA, NARROW>(gu, ctas, st);
    return e == cudaSuccess ? launch_one<Q, 1, ATMA, NARROW>(dn, ctas, st) : e;
}

}  // namespace pair

// The experts' gate/up matrices [E][gate rows, up rows][H] f16 as a 5-D array (input, row of eight, gate | up, group of eight
// rows, expert): a box is 64 inputs of 64 gate and 64 up rows in the order of the pair's operand.
static cudaError_t make_tmap_gate_up(const __half* gu16, int E, int I, int H, CUtensorMap* out) {
    const uint64_t dims[5] = {(uint64_t)H, 8, 2, (uint64_t)I / 8, (uint64_t)E};
    const uint64_t strides[4] = {(uint64_t)H * 2, (uint64_t)I * H * 2, (uint64_t)H * 16, (uint64_t)I * H * 4};
    const uint32_t box[5] = {64, 8, 2, 8, 1};
    return make_tmap_f16_nd(gu16, 5, dims, strides, box, out);
}

// gate/up + SwiGLU, then down. x16: activation rows [columns, H] in the operands' element order, or null: the columns' rows
// are taken from the tokens' plane p.xr16
cudaError_t launch_grouped_pair(const PrefillArgs& p, const void* x16, int tile_cols, int ctas, cudaStream_t st, __half* out16_rows) {
    const bool narrow = tile_cols == pair::Form<true>::cols;
    const int C = p.T * p.K, mt_gu = p.L.I / 128;
    const int max_ct = C / tile_cols + p.L.E;
    pair::Args gu{};
    gu.L = p.L;
    gu.tiles = p.tiles;
    gu.n_tiles = p.n_tiles;
    gu.out16 = p.s16;
    gu.status = p.status;
    gu.status_host = p.status_host;
    gu.wait_limit_ns = p.wait_limit_us ? (uint64_t)p.wait_limit_us * 1000ull : tc::WAIT_LIMIT_NS;
    gu.debug_extra_tx = p.debug_extra_tx;
    gu.kdim = p.L.H;
    gu.out_ld = p.L.I;
    pair::Args dn = gu;
    // the columns are gathered from the tokens' plane, unless they are its rows already (one expert)
    const bool gathered = x16 == nullptr;
    gu.gather = gathered ? p.R.col_src_tok : nullptr;
    gu.n_cols = C;
    dn.debug_extra_tx = 0;  // the hook applies to the first kernel of the pair
    dn.tiles = p.tiles + (size_t)max_ct * mt_gu;  // as laid out by launch_route_large
    dn.out16 = out16_rows ? out16_rows : p.d16;
    dn.out_row_map = out16_rows ? p.R.col_src_tok : nullptr;
    dn.kdim = p.L.I;
    dn.out_ld = p.L.H;
    cudaError_t e = gathered ? make_tmap_f16(p.xr16, (uint64_t)p.T, (uint64_t)p.L.H, 1, &gu.tmap_n)
                             : make_tmap_f16(x16, (uint64_t)C, (uint64_t)p.L.H, 32, &gu.tmap_n);
    if (e == cudaSuccess && !gathered) e = make_tmap_f16(x16, (uint64_t)C, (uint64_t)p.L.H, 128, &gu.tmap_w);
    if (e == cudaSuccess) {
        const uint64_t dims[2] = {(uint64_t)p.L.H, (uint64_t)C}, strides[1] = {(uint64_t)p.L.H * 2};
        const uint32_t box[2] = {32, 32};
        e = make_tmap_f16_nd(p.d16, 2, dims, strides, box, &dn.tmap_o, CU_TENSOR_MAP_SWIZZLE_64B);
    }
    if (e == cudaSuccess) e = make_tmap_f16(p.s16, (uint64_t)C, (uint64_t)p.L.I, 32, &dn.tmap_n);
    if (e == cudaSuccess) e = make_tmap_f16(p.s16, (uint64_t)C, (uint64_t)p.L.I, 128, &dn.tmap_w);
    if (e != cudaSuccess) return e;
    if (p.L.gu16 != nullptr) {
        e = make_tmap_gate_up(p.L.gu16, p.L.E, p.L.I, p.L.H, &gu.tmap_a);
        if (e == cudaSuccess) e = make_tmap_f16(p.L.dn16, (uint64_t)p.L.E * p.L.H, (uint64_t)p.L.I, 128, &dn.tmap_a);
        if (e != cudaSuccess) return e;
        return narrow ? pair::launch_both<BF16, true, true>(gu, dn, ctas, st) : pair::launch_both<BF16, true, false>(gu, dn, ctas, st);
    }
    switch (p.L.quant) {
        case Q4_0: return narrow ? pair::launch_both<Q4_0, false, true>(gu, dn, ctas, st) : pair::launch_both<Q4_0, false, false>(gu, dn, ctas, st);
        case Q8_0: return narrow ? pair::launch_both<Q8_0, false, true>(gu, dn, ctas, st) : pair::launch_both<Q8_0, false, false>(gu, dn, ctas, st);
        default:
            return cudaErrorInvalidValue;  // BF16 layers always carry their f16 matrices on this path
    }
}

}  // namespace lumen
