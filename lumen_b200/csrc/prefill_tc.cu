// Prefill grouped expert products on the 5th-generation tensor cores (tcgen05,
// accumulators in TMEM), one CTA a tile: for expert-parallel calls, and where the grid is capped at one CTA (all other
// calls: prefill_pair.cu). Replaces the reference's tiled prefill kernels
// (moe_grouped_gate_up_swiglu_q4_0_tiled_f32act / moe_grouped_down_q4_0_tiled_f32act,
// cuda/shaders/moe_grouped.cu:1202-1510; the Q8_0 dp4a / mma.sync variants :566-1170,
// :2183-2598; the BF16 variants :1523-1760).
//
// Formulation. Gate/up + SwiGLU ("weights are the M operand"): for a tile of up to 256
// compact columns of one expert,  D_g[128 gate rows, N] += G[128, k] X[N, k]^T  and the
// same for the up rows, two tcgen05.mma of shape M=128 x N(16..256) x K=16 per 16 inputs
// sharing the activation operand; N follows the ragged per-expert column counts
// (Zipf-skewed loads) without padding M. Down ("tokens are the M operand"): for up to 128
// columns,  D[128 tokens, 256 output rows] += S[128, k] W[256, k]^T, one MMA per 16 inputs
// whose N operand is the stage's two adjacent 128-row weight tiles, so that an epilogue
// thread owns one token and stores 32 bytes at a time; a tile of up to 256 columns (a grid capped at one CTA) is two such
// products against the same weight stage, into the two accumulator sets.
//
// One CTA per SM, persistent over a device-built tile list, warp-specialised (27 warps):
//   warps 0-7   epilogue: tcgen05.ld of the accumulators, SwiGLU (gate/up), f16 stores
//               (into another rank's return buffer for an expert-parallel down product)
//   warps 8-23  weight producers, one 16-row tile each per 128-input group: 128-bit loads of
//               the repacked quant tiles (the next group prefetched in registers), dequantise
//               to f16 (scale folded in) in registers, store into the 128-byte-swizzled
//               K-major operand tile in shared memory. When the weights are plain f16
//               matrices copied by TMA (BF16 layers; LUMEN_MOE_FLAG_PREFILL_F16_WEIGHTS) they
//               share the gate/up epilogue instead
//   warp 24     one thread feeds the activation operand (and TMA-fed weights) with
//               cp.async.bulk.tensor.2d boxes of 64 inputs x 32 or 128 rows
//   warp 25     an elected lane issues tcgen05.mma / tcgen05.commit
//   warp 26     one thread hands out the tiles: the CTA's first tile is its index, every further
//               one is claimed from a device-wide counter while the tile before it is being
//               multiplied, and reaches the roles through a small ring of descriptors
// Stages are handed over with mbarriers; every wait is bounded (on expiry the
// kernel raises a status word, drains and frees its TMEM instead of hanging).
//
// Inputs are 16-bit: activations pre-converted to f16 and
// pre-permuted within each 32-block to the order the dequantiser emits (route_tc.cu; natural order for TMA-fed
// weights), gathered into compact-column order (gather_rows_kernel); the SwiGLU output is
// written in the same order so the down product reads it back without any shuffle.
#include "tc_weights.cuh"
#include <type_traits>

namespace lumen {

namespace tc {

constexpr int EPI_WARPS = 8, A_WARPS = 16, B_WARPS = 1;  // B: one thread drives the TMA
constexpr int A_WARP0 = EPI_WARPS, B_WARP0 = A_WARP0 + A_WARPS, MMA_WARP = B_WARP0 + B_WARPS;
constexpr int SCHED_WARP = MMA_WARP + 1;  // one thread hands out the tiles
constexpr int THREADS = (SCHED_WARP + 1) * 32;
// rows of an activation box: 32 where tiles are narrow (no more of the operand is copied than the tile has)
__host__ __device__ constexpr int bbox_rows(int bn) { return bn == 256 ? 128 : 32; }
constexpr int SCHED_RING = 4;             // tile descriptors in flight between the scheduler and the roles

// Position of element e (0..31) of a block in the permuted 16-bit layout:
// chunk t = (e mod 16) / 4, slot order (4t, 4t+2, 16+4t, 16+4t+2, 4t+1, 4t+3, 16+4t+1, 16+4t+3).
__host__ __device__ __forceinline__ int perm_pos(int e) {
    const int hi = e >> 4, r = e & 15, t = r >> 2, m = r & 3;
    const int slot = ((m & 1) ? 4 : 0) + (hi ? 2 : 0) + ((m >> 1) & 1);
    return t * 8 + slot;
}

struct Args {
    CUtensorMap tmap;            // activation operand [rows, kdim] f16, box 64 x 32 or 128, SWIZZLE_128B (first: 64-byte aligned)
    CUtensorMap tmap_a;          // ATMA form: the experts' plain f16 matrices as one 2-D array [E * a_rows_exp, kdim]
    int a_rows_exp;              // rows per expert there: 2 I (gate rows then up rows) or H (down)
    int a_row1;                  // second operand's rows relative to the first: I (up) or 128 (next row tile of down)
    LayerDev L;
    const int4* tiles;
    int32_t* n_tiles;            // [0..1] tiles of the gate/up and the down list, [2..3] the kernels' tile counters (zero at launch)
    __half* out16;          // gate/up: S16 [C, I] permuted order; down: D16 [C, H] natural order
    int32_t* status;
    int32_t* status_host;   // mapped pinned copy of the status word for the host (null = none)
    uint64_t wait_limit_ns; // limit of every mbarrier wait
    int debug_extra_tx;     // test hook: the first stage's barrier expects this many bytes too many
    int kdim;               // H (gate/up) or I (down)
    int out_ld;             // I or H
    const int32_t* out_row_map;  // down mode: output row of compact column c (null = c itself)
    TcPeerOut peer;              // down mode, expert parallel: output rows go to other ranks' buffers (ret_map null = off)
};

// Lane constants of the dequantiser: where a lane's 16-byte chunks go in the operand tile.
// Lanes with odd g handle the second block of a pair first: the eight lanes of a quarter
// warp then hit eight different 16-byte chunk positions (rows are 128 bytes apart, i.e. a
// whole bank cycle) and the 128-bit stores are conflict-free.
template <int Q>
struct DequantLane {
    uint32_t off[2];   // first / second pass, row g (row g + 8 is 1024 bytes on: the same chunk of the swizzle)
    uint32_t bsel[2];  // byte selector of the pass's block scale, in both halves
    bool odd;
    UnpackConst k = unpack_const_pinned<Q>();
    __device__ __forceinline__ DequantLane(int rtl, int lane) {
        const int g = lane >> 2, t = lane & 3;
        odd = (g & 1) != 0;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int second = p ^ (g & 1);
            off[p] = (uint32_t)((rtl * 16 + g) * 128 + ((((second << 2) + t) ^ g) << 4));
            bsel[p] = second ? 0x3232u : 0x1010u;
        }
    }
};

// Dequantise one lane's share of half a weight tile (16 rows x 64 k: blocks 2*sub and 2*sub+1) into the
// operand tile at a_base: 4 chunks of 16 bytes (rows g, g+8). (Beside store_weights: 1 select, 1 scale permute per 8 weights.) The
// arithmetic is that of store_weights, to the bit, written out: through the call, Q8_0 tiles of 128 columns are scheduled worse, with the same registers
// (one expert-parallel rank, 2048 x 768, E = 128, 300 tokens 234.6 -> 237.8 us, 1200 tokens 284.9 -> 287.3).
template <int Q>
__device__ __forceinline__ void dequant_store(const WTile<Q>& w, int sub, uint32_t a_base, const DequantLane<Q>& dl) {
    if constexpr (Q == BF16) return;  // BF16 layers feed this path from plain f16 matrices (ATMA): no producers
    const uint32_t s_g = (sub == 0) ? w.s.x : w.s.y;   // f16 scales of blocks 2 sub, 2 sub + 1: row g
    const uint32_t s_g8 = (sub == 0) ? w.s.z : w.s.w;  // row g + 8
    uint32_t v0[2][2], v1[2][2];  // [pass][row g | g + 8]: the block's words (Q8_0: elements 0..15 | 16..31)
    if (Q == Q4_0) {
        const uint4 v = w.q[sub];
        v0[0][0] = dl.odd ? v.z : v.x;
        v0[1][0] = dl.odd ? v.x : v.z;
        v0[0][1] = dl.odd ? v.w : v.y;
        v0[1][1] = dl.odd ? v.y : v.w;
    } else {
        const uint4 va = w.q[(2 * sub) % QTraits<Q>::NQ], vb = w.q[(2 * sub + 1) % QTraits<Q>::NQ];
        v0[0][0] = dl.odd ? vb.x : va.x;
        v0[1][0] = dl.odd ? va.x : vb.x;
        v1[0][0] = dl.odd ? vb.y : va.y;
        v1[1][0] = dl.odd ? va.y : vb.y;
        v0[0][1] = dl.odd ? vb.z : va.z;
        v0[1][1] = dl.odd ? va.z : vb.z;
        v1[0][1] = dl.odd ? vb.w : va.w;
        v1[1][1] = dl.odd ? va.w : vb.w;
    }
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t sc = prmt(r ? s_g8 : s_g, 0u, dl.bsel[p]);
            uint32_t l0, l1, h0, h1;
            if (Q == Q4_0) {
                const uint32_t x = v0[p][r], y = x >> 8;
                l0 = hsub2_u32(lop_and_or(x, 0x000F000Fu, dl.k.or_a), dl.k.sub_a);
                h0 = hsub2_u32(lop_and_or(x, 0x00F000F0u, dl.k.or_b), dl.k.sub_b);
                l1 = hsub2_u32(lop_and_or(y, 0x000F000Fu, dl.k.or_a), dl.k.sub_a);
                h1 = hsub2_u32(lop_and_or(y, 0x00F000F0u, dl.k.or_b), dl.k.sub_b);
            } else {
                const uint32_t x = v0[p][r] ^ dl.k.or_b, y = v1[p][r] ^ dl.k.or_b;
                l0 = hsub2_u32(prmt(x, dl.k.or_a, 0x4240u), dl.k.sub_a);
                l1 = hsub2_u32(prmt(x, dl.k.or_a, 0x4341u), dl.k.sub_a);
                h0 = hsub2_u32(prmt(y, dl.k.or_a, 0x4240u), dl.k.sub_a);
                h1 = hsub2_u32(prmt(y, dl.k.or_a, 0x4341u), dl.k.sub_a);
            }
            sts128(a_base + dl.off[p] + r * 1024, hmul2_u32(l0, sc), hmul2_u32(h0, sc), hmul2_u32(l1, sc), hmul2_u32(h1, sc));
        }
}

// ATMA: the weight operands are not dequantised here but copied by TMA from plain f16 matrices
// (BF16 layers; Q4_0 / Q8_0 layers of a context created with LUMEN_MOE_FLAG_PREFILL_F16_WEIGHTS): the
// producer warps have nothing to dequantise and every operand is in the natural input order.
//
// Operand stages. The dequantising producers prefetch the next 128-input group of quantised tiles
// into registers while they work on the current one: with sixteen producer warps of one tile
// each that is 3 (Q4_0) or 5 (Q8_0) uint4 per lane in flight, inside the 72 registers a thread has.
// (With eight warps of two tiles the Q8_0 prefetch spilled and a cp.async ring in shared memory
// replaced it, at the price of an operand stage; the ring is gone again: 0.540 -> 0.50 ms per
// 4096-token Q8_0 call.)
// STG (expert-parallel down product): an operand stage is given up for a staging tile from which
// the output rows leave as 256-byte bulk copies (see the epilogue).
template <int Q, int BN, bool ATMA, bool STG = false>
struct StagesOf {
    static constexpr bool ring = (BN == 128) && !ATMA && !STG;
    static constexpr int value = ((BN == 128) ? 4 : 3) - ((STG || ring) ? 1 : 0);
};
// Raw weight ring (128-column tiles, dequantised weights). A tile of few columns has little work
// for the tensor cores, and the register prefetch keeps only one 128-input group (18 KB per SM for
// Q4_0) on the way. Each producer warp therefore owns a ring of RING of its 16-row tiles in
// shared memory, filled by bulk copies (quants and scales of a group are contiguous) that run
// ahead of the dequantisation, across tile boundaries; an operand stage pays for it.
// The 256-column form keeps the register prefetch: its MMAs take longer than the latency.
template <int Q, int BN, bool ATMA, bool STG = false>
struct RingOf {
    static constexpr int value = !StagesOf<Q, BN, ATMA, STG>::ring ? 0 : (Q == Q4_0) ? 4 : 2;
};
template <int Q>
struct RawTile {  // bytes of one 16-row x 128-input tile: quants, then scales
    static constexpr int q_bytes = QTraits<Q>::NQ * 512, bytes = q_bytes + 128;
};
constexpr int STG_ROW_BYTES = 256 + 16;                 // 128 f16 outputs of one token + padding (bank spread)
constexpr int STG_BYTES = 2 * 128 * STG_ROW_BYTES;      // two warp groups x 128 tokens

// Debug aid (compile with -DLUMEN_TC_TRACE): per CTA, the MMA warp's cycles: [2] waiting for full stages, [3] waiting for a
// free accumulator, [4] in all, and [5] its tiles, read back with lumen_debug_tc_trace.
#ifdef LUMEN_TC_TRACE
__device__ unsigned long long g_tc_trace[2][160][8];
#define TRACE_WAIT(acc, expr) ([&] { const long long t0_ = clock64(); const bool r_ = (expr); (acc) += clock64() - t0_; return r_; }())
#define TRACE_PUT(slot, v) g_tc_trace[MODE][blockIdx.x][slot] = (unsigned long long)(v)
#else
#define TRACE_WAIT(acc, expr) (expr)
#define TRACE_PUT(slot, v)
#endif

template <int Q, int MODE, int BN, bool ATMA = false, bool STG = false>
__global__ void __launch_bounds__(THREADS, 1)
grouped_gemm_tc_kernel(const __grid_constant__ Args a) {
    static_assert(!STG || (MODE == 1 && BN == 128), "the staged epilogue belongs to the 128-token down product");
    // Two 128-row weight operands share every activation stage (gate and up rows of the
    // same I range; two adjacent row tiles of the down matrix): the activation operand,
    // which comes from L2 at 2 bytes per element, is then read at half the rate.
    // 256-column tiles (experts of more than 128 columns on average; down: not in an expert-parallel call): each dequantised
    // weight tile serves 256 columns, and with K = H the main loop is long; the two 256-column f32
    // accumulators of a full tile fill TMEM (512 columns), so its epilogue is not overlapped with
    // the next tile's MMAs (its producers do run ahead).
    // 128-column tiles (down: K = I is short, 12 stages at I = 768, so the epilogue weighs
    // more; gate/up of small batches: fewer empty columns): TWO accumulator sets, the
    // epilogue of tile i runs under the MMAs of tile i+1.
    constexpr int NA = 2;
    // BN: columns per tile
    // Accumulator sets in TMEM (512 columns), always two.
    // Down: a set is 256 columns (the output rows of an m-tile) for 128 tokens; a 256-token tile of
    // the BN = 256 form takes both at once (its two token halves, one weight stage serving both),
    // a tile of up to 128 tokens takes one, and the epilogue works through the halves one by one.
    // Gate/up, BN = 128: a set is the gate and the up accumulator side by side (2 x 128 columns).
    // Gate/up, BN = 256: the gate accumulator lives in TMEM columns 0..255 and the up accumulator in
    // 256..511; a tile of up to 128 columns (the last chunk of most experts under skewed loads) takes
    // one HALF of each (set s: columns 128 s.. of both), so two such tiles are in flight and the
    // epilogue of one runs under the MMAs of the next; a wider tile takes both sets at once.
    constexpr int NACC = 2;
    constexpr bool WIDE_GU = (MODE == 0 && BN == 256);
    constexpr int ACC_COLS = WIDE_GU ? 128 : 256;  // TMEM columns from one set to the next
    // While a wide gate/up tile holds both sets the tensor pipe idles during its epilogue. When the weights come
    // by TMA the producer warps have nothing else to do and share the epilogue. (Dequantising
    // producers doing the same was measured slower, 0.52 -> 0.60 ms per 4096-token Q4_0 call: their
    // own work is what those kernels wait for.)
    constexpr bool HELP = WIDE_GU && ATMA;
    constexpr int STAGES = StagesOf<Q, BN, ATMA, STG>::value;  // one stage = 64 inputs (one swizzle atom in K)
    constexpr int STAGE_BYTES = NA * SUB_BYTES + BN * 128;  // A operands then B
    constexpr int TMEM_COLS = 512;
    constexpr int RING = RingOf<Q, BN, ATMA, STG>::value;
    constexpr int BBOX = bbox_rows(BN);

    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full_bar[NACC], acc_empty_bar[NACC];
    __shared__ uint64_t ring_bar[RING ? A_WARPS * RING : 1];
    __shared__ uint32_t tmem_base_s;
    __shared__ uint32_t abort_s;
    // Tiles are handed out dynamically: the CTA's first tile is blockIdx.x, every further one the next
    // of the list not yet taken by any CTA (a device-wide counter). One thread claims a tile while the
    // MMA thread is still inside the tile before it, and passes the descriptor to the roles through
    // this ring. (With tiles dealt round-robin the slowest CTA of a Zipf-loaded 4096-token call ran
    // 11 % longer than the median one in gate/up and 13 % in down.)
    __shared__ int4 sched_tile_s[SCHED_RING];
    __shared__ uint64_t sched_full_bar[SCHED_RING], sched_empty_bar[SCHED_RING], sched_go_bar[2];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t stage0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const AbortCtl abort_flag{&abort_s, a.wait_limit_ns};

    if (tid == 0) {
        abort_s = 0u;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&full_bar[s]), ATMA ? 1 : A_WARPS + 1);  // one arrival per weight-producer warp + the TMA thread's expect_tx
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int b = 0; b < NACC; ++b) {
            mbar_init(smem_u32(&acc_full_bar[b]), 1);
            mbar_init(smem_u32(&acc_empty_bar[b]), HELP ? EPI_WARPS + A_WARPS : EPI_WARPS);
        }
        for (int i = 0; i < A_WARPS * RING; ++i) mbar_init(smem_u32(&ring_bar[i]), 1);
        // readers of a descriptor: epilogue warps, the producer warps when they dequantise or share the
        // epilogue, the TMA thread and the MMA thread
        constexpr int SCHED_READERS = EPI_WARPS + ((!ATMA || HELP) ? A_WARPS : 0) + 2;
        for (int s = 0; s < SCHED_RING; ++s) {
            mbar_init(smem_u32(&sched_full_bar[s]), 1);
            mbar_init(smem_u32(&sched_empty_bar[s]), SCHED_READERS);
        }
        mbar_init(smem_u32(&sched_go_bar[0]), 1);
        mbar_init(smem_u32(&sched_go_bar[1]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                     "r"((uint32_t)TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;

    // (barriers and TMEM are set up above while the kernel before this one may still be running;
    // everything it wrote, the tile list first of all, is read from here on)
    grid_dep_sync();
    const int ntiles = a.n_tiles[MODE];
    const int kgs = a.kdim >> 7;   // 128-input groups (weight tile granularity)
    const int khs = kgs * 2;       // 64-input pipeline stages per tile
    // The n-th tile of this CTA (n counted by the caller): false when the list is exhausted or the
    // kernel gives up. The descriptor is copied and its ring slot released at once. WARP: the whole
    // warp takes it together (one arrival for all lanes), else one thread does.
    auto take_tile = [&](auto warp_tag, int& n, int4& tile) -> bool {
        constexpr bool WARP = decltype(warp_tag)::value;
        const int slot = n % SCHED_RING;
        bool ok = mbar_wait(smem_u32(&sched_full_bar[slot]), (n / SCHED_RING) & 1, abort_flag);
        if constexpr (WARP) ok = __all_sync(0xffffffffu, ok);
        if (!ok) return false;
        tile = sched_tile_s[slot];
        if constexpr (WARP) __syncwarp();
        if (!WARP || lane == 0) mbar_arrive(smem_u32(&sched_empty_bar[slot]));
        ++n;
        return tile.z >= 0;
    };
    auto next_tile = [&](int& n, int4& tile) -> bool { return take_tile(std::false_type{}, n, tile); };
    auto next_tile_warp = [&](int& n, int4& tile) -> bool { return take_tile(std::true_type{}, n, tile); };
    // When the CTA's next tile is claimed: while the MMA warp is in the tile `ahead` before it, at stage go_kh.
    // Long tiles: late in the tile before, so that the last tiles of the list go to the CTAs that are
    // free first, but early enough for the claim (an atomic and a load, ~2 us) to be back when the producers reach
    // the tile's last group. (They take the next descriptor before they fill the last two stages of a
    // tile, so the signal has to come before the MMA warp needs those: go_kh <= khs - 2.)
    // Short tiles (the down product, K = I): a tile is over in about the time of a claim, and the producers' ring would
    // run dry at every tile end; they are claimed two tiles ahead (256 experts, I = 512: 322 -> 250 us per call).
    const int ahead = (khs >= 24) ? 1 : 2;
    const int go_kh = (khs >= 24) ? khs / 2 - 4 : 0;

    // Epilogue of one tile by one warp: the warp's TMEM lanes are 32 (warp % 4).. (hardware rule);
    // of the tile's 16-column TMEM chunks it takes those with chunk % nparts == part.
    auto epilogue_part = [&](const int4& tile, int ab, int h, int part, int nparts) {
        const int row = (warp & 3) * 32 + lane;
        const int ncols = tile.z;
        const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + ab * ACC_COLS;
        if (MODE == 1) {
            // Down product: the tile's columns (tokens) are the TMEM lanes and the 256 output rows
            // of the m-tile the TMEM columns, so a thread owns one token and reads 16 consecutive
            // output rows per load: its stores are 32 bytes wide and each token's 512 bytes are
            // contiguous (a whole NVLink packet when the row lives on another rank).
            {
                const int tcol = h * 128 + row;  // token column of the tile (h: its half of a 256-token tile)
                bool live = tcol < ncols;
                __half* dst = a.out16;
                if (live) {
                    int orow_idx = tile.y + tcol;
                    if (a.out_row_map != nullptr) orow_idx = a.out_row_map[orow_idx];
                    dst = a.out16 + (size_t)orow_idx * a.out_ld;
                    if (a.peer.ret_map != nullptr) {
                        // plain stores into the return buffer of the rank the row came from
                        const int m = a.peer.ret_map[orow_idx];
                        const int pr = (m >> 24) & 0xff, prow = m & 0xffffff;
                        live = pr < a.peer.world && prow < a.peer.rows_cap;  // never leave the buffers
                        if (live) dst = a.peer.base[pr] + (size_t)prow * a.out_ld;
                    }
                    dst += (size_t)tile.w * 256;
                }
                // (every lane takes part in the loads: tcgen05.ld is a warp-wide instruction)
                // a contiguous share of the 256 output rows per warp group
                const int ow = 256 / nparts;
                if constexpr (STG) {
                    // Rows that leave for another GPU: a lane's direct stores are 32-byte pieces of 32
                    // different rows per warp instruction, which cross NVLink as small packets. Here the
                    // lane collects its token's 128 outputs (256 bytes) in shared memory and sends them
                    // as ONE asynchronous bulk copy. Row pitch 272 bytes: the eight lanes of a quarter
                    // warp hit eight different 16-byte bank groups.
                    const uint32_t srow = stage0 + STAGES * STAGE_BYTES + (uint32_t)(part * 128 + row) * STG_ROW_BYTES;
                    // the previous tile's copy of this row must have read its bytes before they are overwritten
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
#pragma unroll 2
                    for (int n0 = 0; n0 < 128; n0 += 16) {
                        uint32_t v[16];
                        tmem_ld16(taddr + part * 128 + n0, v);
                        tmem_ld_wait();
                        uint32_t hh[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const __half2 pr2 = __floats2half2_rn(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                            hh[j] = *reinterpret_cast<const uint32_t*>(&pr2);
                        }
                        sts128(srow + n0 * 2, hh[0], hh[1], hh[2], hh[3]);
                        sts128(srow + n0 * 2 + 16, hh[4], hh[5], hh[6], hh[7]);
                    }
                    fence_proxy_async();  // the lane's own writes, before the async proxy reads them
                    if (live)
                        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], 256;" ::"l"(
                                         __cvta_generic_to_global(dst + part * 128)),
                                     "r"(srow)
                                     : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
                if constexpr (!STG) {
#pragma unroll 2
                for (int n0 = part * ow; n0 < (part + 1) * ow; n0 += 16) {
                    uint32_t v[16];
                    tmem_ld16(taddr + n0, v);
                    tmem_ld_wait();
                    if (live) {
                        uint32_t hh[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const __half2 pr2 = __floats2half2_rn(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                            hh[j] = *reinterpret_cast<const uint32_t*>(&pr2);
                        }
                        st_global_v8(dst + n0, hh);  // 16 outputs = one 32-byte sector of the token's row
                    }
                }
                }
            }
        } else {
            // Gate/up: a thread owns one row of I (its TMEM lane) and walks the token columns
            const int irow = tile.w * 128 + row;  // SwiGLU output is stored in the order the down product reads it
            const size_t off0 = ATMA ? (size_t)irow : (size_t)(irow & ~31) + perm_pos(irow & 31);
            // 8-column pieces of this warp's 16-column chunks, the TMEM loads of the next piece issued
            // before the current one is worked on
            auto piece_col = [&](int p) { return part * 16 + (p >> 1) * nparts * 16 + (p & 1) * 8; };
            __half* const dst0 = a.out16 + (size_t)tile.y * a.out_ld + off0;
            const uint32_t ld = (uint32_t)a.out_ld;
            auto work = [&](int col, const uint32_t (&g)[8], const uint32_t (&u)[8]) {
                __half* dst = dst0 + (size_t)((uint32_t)col * ld);
                if (col + 8 <= ncols) {
#pragma unroll
                    for (int j = 0; j < 8; ++j, dst += ld) *dst = __float2half_rn(swiglu_fast(__uint_as_float(g[j]), __uint_as_float(u[j])));
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j, dst += ld)
                        if (col + j < ncols) *dst = __float2half_rn(swiglu_fast(__uint_as_float(g[j]), __uint_as_float(u[j])));
                }
            };
            uint32_t g0[8], u0[8], g1[8], u1[8];
            int p = 0;
            if (piece_col(0) < ncols) {
                tmem_ld8(taddr + piece_col(0), g0);
                tmem_ld8(taddr + BN + piece_col(0), u0);
            }
            while (piece_col(p) < ncols) {
                // (the loop condition is uniform over the warp: tcgen05.ld is a warp-wide instruction)
                tmem_ld_wait();
                tmem_ld_fence8(g0);
                tmem_ld_fence8(u0);
                const bool more1 = piece_col(p + 1) < ncols;
                if (more1) {
                    tmem_ld8(taddr + piece_col(p + 1), g1);
                    tmem_ld8(taddr + BN + piece_col(p + 1), u1);
                }
                work(piece_col(p), g0, u0);
                if (!more1) break;
                tmem_ld_wait();
                tmem_ld_fence8(g1);
                tmem_ld_fence8(u1);
                if (piece_col(p + 2) < ncols) {
                    tmem_ld8(taddr + piece_col(p + 2), g0);
                    tmem_ld8(taddr + BN + piece_col(p + 2), u0);
                }
                work(piece_col(p + 1), g1, u1);
                p += 2;
            }
        }
    };
    constexpr int EPI_PARTS = EPI_WARPS / 4 + (HELP ? A_WARPS / 4 : 0);  // groups of four warps sharing a tile's epilogue
    // A warp's share of one tile's epilogue. v: accumulator sets handed over so far (set v % NACC, used v / NACC times
    // before). A tile of more than 128 columns holds both sets: the down product works
    // through them one after the other (its two token halves), gate/up reads them as one tile.
    auto epilogue_tile = [&](const int4& tile, int& v, int part) -> bool {
        const int nsets = (tile.z > 128) ? 2 : 1;
        const int passes = (MODE == 1) ? nsets : 1, per_pass = (MODE == 1) ? 1 : nsets;
        for (int h = 0; h < passes; ++h) {
            for (int j = 0; j < per_pass; ++j)
                if (!mbar_wait(smem_u32(&acc_full_bar[(v + j) % NACC]), ((v + j) / NACC) & 1, abort_flag)) return false;
            tc_fence_after();
            epilogue_part(tile, per_pass == 2 ? 0 : v % NACC, h, part, EPI_PARTS);
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
                for (int j = 0; j < per_pass; ++j) mbar_arrive(smem_u32(&acc_empty_bar[(v + j) % NACC]));
            v += per_pass;
        }
        return true;
    };

    if (warp < EPI_WARPS) {
        // ------------------------------ epilogue ------------------------------
        int v = 0;  // accumulator sets handed over so far: set v % NACC, used v / NACC times before
        bool ok = true;
        int tn = 0;
        int4 tile;
        while (ok && next_tile_warp(tn, tile)) ok = epilogue_tile(tile, v, warp >> 2);
        if constexpr (STG) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // every row has been written
    } else if (warp < B_WARP0) {
        // --------------------------- weight producers --------------------------
        // Sixteen warps, one 16-row weight tile each per 128-input group: warps 0-7 the eight row
        // tiles of the stage's first operand, warps 8-15 those of the second.
        const int pw = warp - A_WARP0;
        const int op = pw >> 3, rtl = pw & 7;  // operand of the stage, 16-row tile within its 128 rows
        bool ok = true;
        int tn = 0;
        // quant words and scales of this warp's tile of 128-input group kg of a tile of the list
        auto tile_ptrs = [&](const int4& tile, int kg, const uint4*& qp, const uint4*& sp) {
            const int e = tile.x;
            int tidx;
            const uint4 *qb, *sb;
            if (MODE == 0) {
                // m-tile = 128 rows of I: operand 0 gate, operand 1 up
                qb = op ? a.L.up_q(e) : a.L.gate_q(e);
                sb = op ? a.L.up_s(e) : a.L.gate_s(e);
                tidx = (tile.w * 8 + rtl) * kgs + kg;
            } else {
                // m-tile = 256 rows of H: two adjacent 128-row tiles
                qb = a.L.down_q(e);
                sb = a.L.down_s(e);
                tidx = (tile.w * 16 + pw) * kgs + kg;
            }
            qp = qb + ((size_t)tidx * QTraits<Q>::NQ) * 32;
            sp = sb + (size_t)tidx * 8;
        };
        auto warp_wait = [&](uint32_t bar, uint32_t parity) -> bool { return mbar_wait(bar, parity, abort_flag); };
        auto warp_arrive = [&](uint32_t bar) {
            fence_proxy_async();  // every lane's own stores, before the warp's one arrival
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };
        const DequantLane<Q> dl(rtl, lane);
        int s = 0, ph = 0;  // operand stage and its parity
        // one half tile into the next stage
        auto produce = [&](const WTile<Q>& w, int sub) -> bool {
            const bool r = __all_sync(0xffffffffu, warp_wait(smem_u32(&empty_bar[s]), ph ^ 1));
            if (r) {
                dequant_store<Q>(w, sub, stage0 + s * STAGE_BYTES + op * SUB_BYTES, dl);
                warp_arrive(smem_u32(&full_bar[s]));
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1;
                }
            }
            return r;
        };
        if constexpr (RING > 0) {
            // Groups flow through this warp's ring in the order of the tile list: `issued` counts the
            // groups requested, `taken` those copied to registers; a slot is refilled as soon as its
            // words are in registers. The descriptor of the CTA's next tile is taken only when it is
            // there already (or when nothing is left to do): waiting for it with groups of the current
            // tile undone would wait for the MMA warp, which waits for those groups.
            constexpr uint32_t RAW = RawTile<Q>::bytes, RAW_Q = RawTile<Q>::q_bytes;
            const uint32_t ring0 = stage0 + STAGES * STAGE_BYTES + (uint32_t)pw * RING * RAW;
            const uint32_t bar0 = smem_u32(&ring_bar[pw * RING]);
            int4 tile = make_int4(0, 0, -1, 0);
            int issued = 0, taken = 0, pkg = kgs;
            bool more = true;  // the list may hold further tiles
            const uint4 *qp = nullptr, *sp = nullptr;
            auto top_up = [&]() {
                while (issued - taken < RING) {
                    if (pkg == kgs) {
                        if (!more) return;
                        if (issued != taken) {
                            const int slot = tn % SCHED_RING;
                            const bool there = mbar_try(smem_u32(&sched_full_bar[slot]), (tn / SCHED_RING) & 1);
                            if (!__all_sync(0xffffffffu, there)) return;
                        }
                        more = next_tile_warp(tn, tile);
                        if (!more) return;
                        pkg = 0;
                        tile_ptrs(tile, 0, qp, sp);
                    }
                    if (elect_one()) {
                        const int slot = issued % RING;
                        const uint32_t bar = bar0 + slot * 8, dst = ring0 + slot * RAW;
                        mbar_expect_tx(bar, RAW);
                        bulk_load(dst, qp, RAW_Q, bar);
                        bulk_load(dst + RAW_Q, sp, RAW - RAW_Q, bar);
                    }
                    __syncwarp();
                    qp += RAW_Q / 16;
                    sp += 8;
                    ++issued;
                    ++pkg;
                }
            };
            top_up();
            while (ok && issued != taken) {
                const int slot = taken % RING;
                ok = __all_sync(0xffffffffu, warp_wait(bar0 + slot * 8, (taken / RING) & 1));
                if (!ok) break;
                WTile<Q> cur;
                const uint32_t src = ring0 + slot * RAW;
#pragma unroll
                for (int j = 0; j < QTraits<Q>::NQ; ++j) cur.q[j] = lds128(src + j * 512 + lane * 16);
                cur.s = lds128(src + RAW_Q + (lane >> 2) * 16);
                ++taken;
                // (the slot is refilled behind the first half's proxy fence and warp barrier: every lane's reads of
                // it are then ordered before the bulk copy's writes)
                ok = produce(cur, 0);
                if (!ok) break;
                top_up();
                ok = produce(cur, 1);
            }
            // give-up: the copies still in flight land before the shared memory goes away
            for (; taken != issued; ++taken)
                for (int i = 0; i < (1 << 16) && !mbar_try(bar0 + (taken % RING) * 8, (taken / RING) & 1); ++i) {}
        } else if constexpr (!ATMA) {
            WTile<Q> cur, nxt;
            auto issue = [&](const int4& tile, int kg, WTile<Q>& dst) {
                const uint4 *qp, *sp;
                tile_ptrs(tile, kg, qp, sp);
    #pragma unroll
                for (int j = 0; j < QTraits<Q>::NQ; ++j) dst.q[j] = ldg_stream(qp + j * 32 + lane);
                if (Q != BF16) dst.s = ldg_stream(sp + (lane >> 2));
            };
            // The next tile's descriptor is taken before the last group of the current tile, so that
            // the first group of the next tile is in flight while the last one is dequantised.
            int4 tile_c, tile_n = make_int4(0, 0, -1, 0);
            bool have_c = next_tile_warp(tn, tile_c), have_n = false;
            if (have_c) issue(tile_c, 0, cur);
            int kg = 0;
            while (ok && have_c) {
                bool more = true;  // a group follows this one
                if (kg + 1 < kgs) {
                    issue(tile_c, kg + 1, nxt);
                } else {
                    have_n = next_tile_warp(tn, tile_n);
                    if (have_n) issue(tile_n, 0, nxt);
                    more = have_n;
                }
                ok = produce(cur, 0) && produce(cur, 1);
                if (more) cur = nxt;
                if (++kg == kgs) {
                    kg = 0;
                    tile_c = tile_n;
                    have_c = have_n;
                    have_n = false;
                }
            }
        }
        if constexpr (HELP) {
            // TMA-fed weights, one accumulator set: nothing to dequantise, the warp takes a share of
            // every tile's epilogue instead
            int4 tile;
            int v = 0;
            while (ok && next_tile_warp(tn, tile)) ok = epilogue_tile(tile, v, EPI_WARPS / 4 + (pw >> 2));
        }
        (void)warp_wait;
        (void)warp_arrive;
        (void)tile_ptrs;
        (void)produce;
    } else if (warp < MMA_WARP) {
        // ------------------------- activation producers ------------------------
        // One thread feeds the activation operand with TMA: per 64-input stage one or two
        // 128-row boxes of the compact (pre-gathered, pre-permuted) f16 activations land
        // in the SWIZZLE_128B layout the MMA descriptor expects; completion is counted in
        // bytes on the stage's full barrier.
        if (lane == 0) {
            const uint64_t tmap_addr = reinterpret_cast<uint64_t>(&a.tmap);
            const uint64_t tmap_a_addr = reinterpret_cast<uint64_t>(&a.tmap_a);
            int row0 = 0, nbox = 1, arow0 = 0;
            bool ok = true;
            int tn = 0, n = 0;
            for (; ok; ++n) {
                const int kh = n % khs;
                if (kh == 0) {
                    int4 tile;
                    if (!next_tile(tn, tile)) break;
                    row0 = tile.y;
                    nbox = (tile.z + BBOX - 1) / BBOX;
                    arow0 = tile.x * a.a_rows_exp + tile.w * (MODE == 0 ? 128 : 256);
                }
                const int s = n % STAGES, ph = (n / STAGES) & 1;
                ok = mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1, abort_flag);
                if (!ok) break;
                const uint32_t bar = smem_u32(&full_bar[s]);
                const uint32_t bbase = stage0 + s * STAGE_BYTES + NA * SUB_BYTES;
                // (test hook: with debug_extra_tx the very first stage can never complete)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                             "r"(nbox * BBOX * 128 + (ATMA ? NA : 0) * SUB_BYTES + (n == 0 ? a.debug_extra_tx : 0))
                             : "memory");
                if (ATMA) {
#pragma unroll
                    for (int op = 0; op < NA; ++op)
                        asm volatile(
                            "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
                            "[%0], [%1, {%2, %3}], [%4];" ::"r"(stage0 + s * STAGE_BYTES + op * SUB_BYTES),
                            "l"(tmap_a_addr), "r"(kh * 64), "r"(arow0 + op * a.a_row1), "r"(bar)
                            : "memory");
                }
                for (int q = 0; q < nbox; ++q)
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
                        "[%0], [%1, {%2, %3}], [%4];" ::"r"(bbase + q * BBOX * 128),
                        "l"(tmap_addr), "r"(kh * 64), "r"(row0 + q * BBOX), "r"(bar)
                        : "memory");
            }
            if (*abort_flag.flag) let_land(smem_u32(&full_bar[0]), STAGES, n);
        }
        __syncwarp();
    } else if (warp == MMA_WARP) {
        // -------------------------------- MMA ---------------------------------
        {
            int tl = 0, s = 0, ph = 0;  // operand stage and its parity
            bool ok = true;
            long long tr_wf = 0, tr_wa = 0;
            const long long tr_t0 = clock64();
            int v = 0;  // accumulator sets taken so far (see the epilogue)
            int tn = 0;
            int4 tile;
            for (; ok && next_tile_warp(tn, tile); ++tl) {
                const int n16 = (tile.z + 15) & ~15;
                // down: D[128 tokens, 256 output rows] = X[128, k] W[256, k]^T, the two adjacent 128-row
                // weight operands of a stage forming one 256-row N operand; a tile of more than 128
                // tokens is two such products per 16 inputs, into two accumulator sets
                const uint32_t idesc = make_idesc(MODE == 1 ? 256 : n16, false);  // (every operand is f16)
                const int nh = (tile.z > 128) ? 2 : 1;  // accumulator sets of the tile
                for (int h = 0; ok && h < nh; ++h) {
                    const int ab = (v + h) % NACC, use = (v + h) / NACC;
                    ok = TRACE_WAIT(tr_wa, mbar_wait(smem_u32(&acc_empty_bar[ab]), (use & 1) ^ 1, abort_flag));
                }
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                const uint32_t acc0 = tmem_base + (v % NACC) * ACC_COLS, acc1 = tmem_base + ((v + 1) % NACC) * ACC_COLS;
                for (int kh = 0; kh < khs; ++kh) {
                    if (kh == go_kh && lane == 0) mbar_arrive(smem_u32(&sched_go_bar[tl % ahead]));  // the CTA's next tile may be claimed now
                    ok = __all_sync(0xffffffffu, TRACE_WAIT(tr_wf, mbar_wait(smem_u32(&full_bar[s]), ph, abort_flag)));
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint64_t w0 = make_desc(stage0 + s * STAGE_BYTES), b0 = w0 + (NA * SUB_BYTES >> 4);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const uint32_t acc = (kh > 0 || j > 0) ? 1u : 0u;
                            if (MODE == 1) {
                                umma(acc0, b0 + j * 2, w0 + j * 2, idesc, acc);
                                if (BN == 256 && nh == 2) umma(acc1, b0 + (SUB_BYTES >> 4) + j * 2, w0 + j * 2, idesc, acc);
                            } else {
#pragma unroll
                                for (int op = 0; op < NA; ++op)
                                    umma((nh == 2 ? tmem_base : acc0) + op * BN, w0 + op * (SUB_BYTES >> 4) + j * 2, b0 + j * 2,
                                         idesc, acc);
                            }
                        }
                        umma_commit(smem_u32(&empty_bar[s]));
                        if (kh == khs - 1)
                            for (int h = 0; h < nh; ++h) umma_commit(smem_u32(&acc_full_bar[(v + h) % NACC]));
                    }
                    __syncwarp();
                    if (++s == STAGES) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (!ok) break;
                v += nh;
            }
            if (lane == 0) {
                TRACE_PUT(2, tr_wf);
                TRACE_PUT(3, tr_wa);
                TRACE_PUT(4, clock64() - tr_t0);
                TRACE_PUT(5, tl);
            }
            (void)tr_wf;
            (void)tr_wa;
            (void)tr_t0;
        }
        __syncwarp();
    } else {
        // ------------------------------ scheduler ------------------------------
        if (lane == 0) {
            for (int n = 0;; ++n) {
                const int slot = n % SCHED_RING;
                // tile n is claimed once the MMA warp is far enough into tile n - ahead (one barrier per parity
                // of that tile when ahead = 2: the warp cannot come round to the same barrier before this wait is over,
                // because tile n is not handed out before it)
                const int m = n - ahead;
                if (m >= 0 && !mbar_wait(smem_u32(&sched_go_bar[m % ahead]), (m / ahead) & 1, abort_flag)) break;
                if (!mbar_wait(smem_u32(&sched_empty_bar[slot]), ((n / SCHED_RING) & 1) ^ 1, abort_flag)) break;
                // the first `ahead` tiles are the CTA's by its index
                const int t = (n < ahead) ? (int)blockIdx.x + n * (int)gridDim.x : ahead * (int)gridDim.x + atomicAdd(a.n_tiles + 2 + MODE, 1);
                sched_tile_s[slot] = (t < ntiles) ? a.tiles[t] : make_int4(0, 0, -1, 0);  // columns < 0: no more tiles
                mbar_arrive(smem_u32(&sched_full_bar[slot]));
                if (t >= ntiles) break;
            }
        }
        __syncwarp();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS)
                     : "memory");
    }
    if (tid == 0 && abort_s) raise_status(a.status, a.status_host, 4);  // LUMEN_MOE_TIMEOUT
}

// rows of the activations' high plane (f16, already in the operand's element order) in compact-column order (row c =
// token col_src_tok[c]): the grouped GEMM then reads plain 2-D boxes of it with TMA. Bound by its writes; eight rows per CTA
// step, their source rows known first and all loads of a thread in flight together. (Converting from the caller's
// f32 rows here instead, after the router's pre-pass had done it already, took 89 us at 8192 tokens, H = 2048, against
// 50.)
__global__ void __launch_bounds__(256)
gather_rows_kernel(const uint4* __restrict__ plane, const int32_t* __restrict__ col_src_tok, int C, int H8, uint4* __restrict__ out) {
    grid_dep_sync();
    constexpr int R = 8;
    const int c0 = blockIdx.x * R;
    int tok[R];
#pragma unroll
    for (int r = 0; r < R; ++r) tok[r] = col_src_tok[min(c0 + r, C - 1)];
    for (int i = threadIdx.x; i < H8; i += 256) {
        uint4 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = __ldg(plane + (size_t)tok[r] * H8 + i);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (c0 + r < C) out[(size_t)(c0 + r) * H8 + i] = v[r];
    }
}

}  // namespace tc

cudaError_t launch_gather_rows(const __half* plane, const int32_t* col_src_tok, int C, int H, void* out, cudaStream_t st) {
    count_launch();
    return launch_dep(tc::gather_rows_kernel, dim3((C + 7) / 8), dim3(256), 0, st, reinterpret_cast<const uint4*>(plane), col_src_tok, C,
                      H / 8, reinterpret_cast<uint4*>(out));
}

cudaError_t make_tmap_f16_nd(const void* base, int nd, const uint64_t* dims, const uint64_t* strides, const uint32_t* box, CUtensorMap* out, CUtensorMapSwizzle swizzle) {
    typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static EncodeFn encode = nullptr;
    if (!encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres);
        if (e != cudaSuccess) return e;
        if (qres != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
        encode = reinterpret_cast<EncodeFn>(fn);
    }
    cuuint64_t d[5], st[4];
    cuuint32_t bx[5];
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    for (int i = 0; i < nd; ++i) {
        d[i] = dims[i];
        bx[i] = box[i];
        if (i + 1 < nd) st[i] = strides[i];
    }
    const CUresult r = encode(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, (cuuint32_t)nd, const_cast<void*>(base), d, st, bx, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t make_tmap_f16(const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows, CUtensorMap* out) {
    const uint64_t dims[2] = {cols, rows}, strides[1] = {cols * 2};
    const uint32_t box[2] = {64, box_rows};
    return make_tmap_f16_nd(base, 2, dims, strides, box, out);
}

template <int Q, int MODE, int BN, bool ATMA = false, bool STG = false>
static cudaError_t launch_tc_one(const tc::Args& a, int grid, cudaStream_t st) {
    constexpr int NA = 2;
    constexpr int STAGES = tc::StagesOf<Q, BN, ATMA, STG>::value;
    const int smem = STAGES * (NA * tc::SUB_BYTES + BN * 128) + 1024 + (STG ? tc::STG_BYTES : 0) +
                     tc::A_WARPS * tc::RingOf<Q, BN, ATMA, STG>::value * tc::RawTile<Q>::bytes;
    static SmemOptIn optin;
    {
        cudaError_t e = ensure_dyn_smem(tc::grouped_gemm_tc_kernel<Q, MODE, BN, ATMA, STG>, (size_t)smem, optin);
        if (e != cudaSuccess) return e;
    }
    count_launch();
    return launch_dep(tc::grouped_gemm_tc_kernel<Q, MODE, BN, ATMA, STG>, dim3(grid), dim3(tc::THREADS), (size_t)smem, st, a);
}

// gate/up + SwiGLU then down, both on tcgen05. x16: permuted 16-bit activations [T,H].
cudaError_t launch_grouped_tc(const PrefillArgs& p, const void* x16, int grid, cudaStream_t st, __half* out16_rows,
                              const TcPlan& plan, const TcPeerOut* peer) {
    const int C = plan.rows, gu_cols = plan.gu_cols;
    const int max_ct = C / gu_cols + p.L.E;
    // rows that go to other ranks' return buffers leave through the staged epilogue (bulk copies)
    const bool stg = peer != nullptr;
    // down tiles as wide as the gate/up ones, except there: its epilogue stores into other GPUs' memory, and with two
    // independent accumulator sets those stores always run under the next tile's MMAs
    const bool dn256 = gu_cols == 256 && !stg;
    const int mt_gu = p.L.I / 128;
    tc::Args gu{};
    cudaError_t te = make_tmap_f16(x16, (uint64_t)C, (uint64_t)p.L.H, tc::bbox_rows(gu_cols), &gu.tmap);
    if (te != cudaSuccess) return te;
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
    tc::Args dn = gu;
    te = make_tmap_f16(p.s16, (uint64_t)C, (uint64_t)p.L.I, tc::bbox_rows(dn256 ? 256 : 128), &dn.tmap);
    if (te != cudaSuccess) return te;
    dn.debug_extra_tx = 0;  // the hook applies to the first kernel of the pair
    dn.tiles = p.tiles + (size_t)max_ct * (mt_gu > 0 ? mt_gu : 1);  // as laid out by launch_route_large
    // out16_rows: write the down product straight into caller rows (row = col_src_tok[column])
    dn.out16 = out16_rows ? out16_rows : p.d16;
    dn.out_row_map = out16_rows ? p.R.col_src_tok : nullptr;
    if (peer) dn.peer = *peer;
    dn.kdim = p.L.I;
    dn.out_ld = p.L.H;
    cudaError_t e;
    if (p.L.gu16 != nullptr) {
        // TMA-fed weights: the experts' plain f16 matrices as two 2-D arrays
        te = make_tmap_f16(p.L.gu16, (uint64_t)p.L.E * 2 * p.L.I, (uint64_t)p.L.H, 128, &gu.tmap_a);
        if (te != cudaSuccess) return te;
        gu.a_rows_exp = 2 * p.L.I;
        gu.a_row1 = p.L.I;
        te = make_tmap_f16(p.L.dn16, (uint64_t)p.L.E * p.L.H, (uint64_t)p.L.I, 128, &dn.tmap_a);
        if (te != cudaSuccess) return te;
        dn.a_rows_exp = p.L.H;
        dn.a_row1 = 128;
        e = (gu_cols == 256) ? launch_tc_one<BF16, 0, 256, true>(gu, grid, st) : launch_tc_one<BF16, 0, 128, true>(gu, grid, st);
        if (e != cudaSuccess) return e;
        if (stg) return launch_tc_one<BF16, 1, 128, true, true>(dn, grid, st);
        return dn256 ? launch_tc_one<BF16, 1, 256, true>(dn, grid, st) : launch_tc_one<BF16, 1, 128, true>(dn, grid, st);
    }
    switch (p.L.quant) {
        case Q4_0:
            e = (gu_cols == 256) ? launch_tc_one<Q4_0, 0, 256>(gu, grid, st) : launch_tc_one<Q4_0, 0, 128>(gu, grid, st);
            if (e != cudaSuccess) return e;
            if (stg) return launch_tc_one<Q4_0, 1, 128, false, true>(dn, grid, st);
            return dn256 ? launch_tc_one<Q4_0, 1, 256>(dn, grid, st) : launch_tc_one<Q4_0, 1, 128>(dn, grid, st);
        case Q8_0:
            e = (gu_cols == 256) ? launch_tc_one<Q8_0, 0, 256>(gu, grid, st) : launch_tc_one<Q8_0, 0, 128>(gu, grid, st);
            if (e != cudaSuccess) return e;
            if (stg) return launch_tc_one<Q8_0, 1, 128, false, true>(dn, grid, st);
            return dn256 ? launch_tc_one<Q8_0, 1, 256>(dn, grid, st) : launch_tc_one<Q8_0, 1, 128>(dn, grid, st);
        default:
            // BF16 layers always carry their plain f16 matrices on this path (see above)
            return cudaErrorInvalidValue;
    }
}

}  // namespace lumen

#ifdef LUMEN_TC_TRACE
extern "C" __attribute__((visibility("default"))) int lumen_debug_tc_trace(unsigned long long* out) {
    return (int)cudaMemcpyFromSymbol(out, lumen::tc::g_tc_trace, sizeof(unsigned long long) * 2 * 160 * 8);
}
#endif
