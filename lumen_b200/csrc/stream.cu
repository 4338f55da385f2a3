// Expert products for batches in which an expert has few columns (decode batches, short prompts):
// weights streamed once, multiplied on the warp-level tensor cores straight from registers.
//
// With a handful of columns per expert a layer call reads every selected expert's weights (340 MB
// at H=2048, I=768, E=128, Q4_0) for little arithmetic. The tcgen05 kernel (prefill_tc.cu) has
// to write each dequantised weight to shared memory as a rounded f16 operand: ~340 instructions per
// 16 x 128 tile, which is what bounds it there (1.9 TB/s at 77 tokens). Here a
// weight goes from the quant planes to an mma.sync fragment as an exact small integer, the f32 scale is
// applied to the block's sums, and nothing is written back.
//
// A WARP owns an item (16 output rows of one expert times one chunk of its columns, all inputs). Items are
// dealt to the CTAs (one per SM) as contiguous ranges of equal cost, experts outermost, so that the warps of an SM work
// on neighbouring rows of one or two experts and find their activations in L1; inside the range the warps take
// every WARPS-th item; no CTA-wide synchronisation anywhere. (A down kernel with the rows outermost, whose CTAs could combine their rows
// themselves, had every warp on another expert and waited for L2 at each 32-input block: 25 instead of 20 us at
// 16 tokens.) Each warp keeps a ring of its own in flight in shared memory, filled by bulk copies on its own
// mbarriers across item boundaries. (cp.async by all lanes instead: 124 -> 138 us at 77 tokens, 193 -> 201 us for a 13-token
// Q8_0 decode at H = 4096.)
//
//   GATE_UP_1 / DOWN_1    prompts: single f16 activation rows in the planes' element order (x16, s16), the precision
//                         of the tcgen05 path; f16 rows out (moe_grouped.cu:1202-1510); the weighted sum
//                         follows in scatter_accum_kernel
//   GATE_UP_2 / DOWN_2    decode batches: hi + lo fragments, two MMA columns per token; f32 sums out
//   DOWN_2I               the same on the integer tensor cores: Q4_0 nibbles against the two-term int8 SwiGLU blocks of
//                         gate_up_stream_kernel
//   (gate/up: cuda/shaders/moe_expert_q4_0.cu:58-108, moe_expert.cu:47-97; down: moe_expert_q4_0.cu:118-151)
#include "decode_common.cuh"
#include "tc_common.cuh"
#include <type_traits>

namespace lumen {

namespace stream {

using namespace dcommon;

enum Mode { GATE_UP_1, DOWN_1, GATE_UP_2, DOWN_2, DOWN_2I };

// Warps per SM and groups in flight per warp: 131..197 KB on the way per SM (the copy peak times the latency is ~55 KB),
// the rest of the 256 KB is L1 for the activations. An item is a chain (its chunk, its columns, its tiles, its rows out), and
// the warps of an SM end unevenly; more warps with shorter rings help the decode down products, whose items are short (16 warps
// -> now, us a call: 4 tokens of Q8_0, 1408 inputs, 53.1 -> 50.2; 8 tokens of Q4_0, 512 inputs, 40.8 -> 39.1; with 32 warps
// 16 tokens of Q4_0 61.7 -> 66.4), not gate/up, which needs the registers (Q8_0 with 20 warps: 13 tokens, H = 4096, 190 -> 194).
template <int Q, int MODE, int WARPS>
struct Shape {
    static constexpr bool down = (MODE == DOWN_1 || MODE == DOWN_2 || MODE == DOWN_2I), int8 = (MODE == DOWN_2I);
    static constexpr int terms = (MODE == GATE_UP_1 || MODE == DOWN_1) ? 1 : 2;
    static constexpr int nm = down ? 1 : 2;  // matrices of an item: down | gate and up
    static constexpr int grp = (Q == Q4_0) ? 2 : 1;  // 128-input groups of a ring slot
    static constexpr int warps = WARPS, ring = (!down ? (Q == Q4_0 ? 4 : 2) : warps > 16 ? (Q == Q4_0 ? 6 : 3) : (Q == Q4_0 ? 8 : 4)) / grp;
    static constexpr uint32_t q_bytes = QTraits<Q>::NQ * 512, s_bytes = (Q == BF16 ? 0 : 128);  // of a tile: quants, scales
    static constexpr uint32_t tile = grp * (q_bytes + s_bytes);
    static constexpr uint32_t slot = nm * tile;
    static constexpr size_t smem = (size_t)warps * ring * slot;
};
template <int Q, int MODE>
constexpr int default_warps() {
    return Q == BF16 ? 8 : 16;
}

struct Args {
    LayerDev L;
    const int4* chunks;         // {expert, first column, columns, -}, `chunk_stride` entries apart
    int chunk_stride;
    const int32_t* starts;      // [CTAs + 1] first item of every CTA (null: equal shares of n_chunks)
    const int32_t* n_chunks;
    const int32_t* col_src_tok; // gate/up: activation row of a compact column (null = the column itself)
    const uint4* b;             // activation rows: f16 [row][kdim] | fragments [row][2][nblk_pad][4] | int8 blocks [row][sq]
    size_t b_row;               // uint4 per row (TERMS 2: per row and term)
    __half* out16;              // GATE_UP_1: s16 [C, I] (permuted order); DOWN_1: d16 [C, H]
    uint4* sf;                  // GATE_UP_2: SwiGLU fragments
    float* d32;                 // DOWN_2(I): [C, H]
    const int32_t* out_row_map; // DOWN_1: output row of compact column c (null = c itself)
    TcPeerOut peer;             // DOWN_1, expert parallel: output rows go to other ranks' buffers (ret_map null = off)
    int32_t* status;            // the context's status word and its copy for the host
    int32_t* status_host;
    uint32_t wait_limit_ns;     // limit of a warp's wait for a copy of its own
    int debug_extra_tx;         // test hook: the first slot of a CTA's first warp expects this many bytes more than arrive
};

// A lane's wait for one of its warp's copies; false once the limit is over.
__device__ __forceinline__ bool wait_copy(uint32_t bar, uint32_t parity, uint32_t limit_ns) {
    for (uint32_t i = 1, t0 = 0; !tc::mbar_try(bar, parity); ++i) {
        if ((i & 63u) == 0u) {
            const uint32_t t = (uint32_t)tc::globaltimer_ns();
            if (i == 64u) t0 = t;
            else if (t - t0 > limit_ns) return false;
        }
    }
    return true;
}
constexpr uint32_t DRAIN_NS = 1000000;  // a warp that gives up waits this long for each copy still on its way

// b fragments of the block's two MMAs out of one 16-byte chunk (the two layouts order them differently)
template <int TERMS>
__device__ __forceinline__ void b_regs(const uint4& v, uint32_t& l0, uint32_t& l1, uint32_t& h0, uint32_t& h1) {
    l0 = v.x;
    l1 = (TERMS == 1) ? v.z : v.y;
    h0 = (TERMS == 1) ? v.y : v.z;
    h1 = v.w;
}

// acc += scale * (block b of the tile) x (eight columns)
template <int Q, int TERMS>
__device__ __forceinline__ void block_mma(const uint32_t (&lo)[4], const uint32_t (&hi)[4], const float2 sc, const uint4& bv,
                                          float (&acc)[4]) {
    uint32_t l0, l1, h0, h1;
    b_regs<TERMS>(bv, l0, l1, h0, h1);
    if constexpr (Q == BF16) {
        mma_bf16(acc, lo, l0, l1);
        mma_bf16(acc, hi, h0, h1);
    } else {
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        mma_f16(c, lo, l0, l1);
        mma_f16(c, hi, h0, h1);
        acc[0] = fmaf(sc.x, c[0], acc[0]);
        acc[1] = fmaf(sc.x, c[1], acc[1]);
        acc[2] = fmaf(sc.y, c[2], acc[2]);
        acc[3] = fmaf(sc.y, c[3], acc[3]);
    }
}

__device__ __forceinline__ uint32_t h2_bits(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t v) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}

// position of element e of a 32-block in the 16-bit rows (perm_pos of prefill_tc.cu)
__device__ __forceinline__ int perm32(int e) {
    const int hi = e >> 4, r = e & 15, t = r >> 2, m = r & 3;
    return t * 8 + ((m & 1) ? 4 : 0) + (hi ? 2 : 0) + ((m >> 1) & 1);
}

template <int Q, int MODE, int WARPS = default_warps<Q, MODE>()>
__global__ void __launch_bounds__(WARPS * 32, 1)
stream_kernel(const __grid_constant__ Args a) {
    using S = Shape<Q, MODE, WARPS>;
    constexpr bool DOWN = S::down, I8 = S::int8;
    constexpr int RING = S::ring, NM = S::nm, TERMS = S::terms, NQ = QTraits<Q>::NQ, GRP = S::grp;
    static_assert(!I8 || Q == Q4_0, "the integer form is for Q4_0 nibbles");
    static_assert(Q != BF16 || TERMS == 2, "prompts of BF16 layers take the tcgen05 kernels");
    extern __shared__ __align__(128) uint8_t ring_smem[];  // [WARPS][RING][NM][quants of GRP groups | their scales]
    __shared__ uint64_t bar_s[WARPS * RING];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gq = lane >> 2, t4 = lane & 3;
    const uint32_t ring = tc::smem_u32(ring_smem) + (uint32_t)warp * RING * S::slot;
    const uint32_t bar0 = tc::smem_u32(&bar_s[warp * RING]);
    if (lane < RING) tc::mbar_init(bar0 + lane * 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();
    // The chunk list comes from the routing kernels. gate/up follows them directly; its own wait makes them
    // complete before it lets the down kernel start, which may therefore request weights right away.
    if (!DOWN) {
        pdl_wait();
        pdl_trigger();
    }
    const int rt_n = DOWN ? a.L.rt_h : a.L.rt_i, kg_n = DOWN ? a.L.kg_i : a.L.kg_h;
    const int nblk_pad = kg_n * 4;
    int i0, i1;
    if (a.starts != nullptr) {
        i0 = a.starts[blockIdx.x];
        i1 = a.starts[blockIdx.x + 1];
    } else {
        const int total = *a.n_chunks * rt_n;
        i0 = (int)((long long)total * blockIdx.x / gridDim.x);
        i1 = (int)((long long)total * (blockIdx.x + 1) / gridDim.x);
    }

    // Warps that take part where there are more items than warps: in a decode batch of Q4_0, and in the BF16 down product of twelve warps, as many
    // as give each the same number of items, so that the last round is as full as the others (16 tokens of Q4_0 61.1 -> 60.8 us, 8 tokens of
    // H = 4096, I = 1536 108.7 -> 103.5). Elsewhere a warp less on the way costs more than the uneven round (90 tokens of Q8_0 155 -> 163, 110
    // of Q4_0 129 -> 132). With a round or less there is nothing to even out, and the two divisions stand in front of the first request (4 tokens
    // of 512 x 256 15.3 -> 14.5 us, 2 of 3072 x 1024 35.7 -> 35.1).
    int nw = WARPS;
    // (16 warps on int8 are for batches of fewer items, and pay for the code: a lone expert of 1024 x 2816 with 16 tokens 39.3 -> 42.0)
    if (((Q == Q4_0 && TERMS == 2 && !(I8 && WARPS == 16)) || (Q == BF16 && DOWN && WARPS > 8)) && i1 - i0 > WARPS) {
        const int n = i1 - i0, rounds = (n + WARPS - 1) / WARPS;
        nw = (n + rounds - 1) / rounds;
        if (warp >= nw) i1 = i0;
    }
    // request cursor: the next groups (of item pi, from group pkg on) to copy, into ring slot wslot
    int pi = i0 + warp, pkg = 0, wslot = 0, rslot = 0;
    uint32_t rphase = 0;
    const uint4 *pq[NM], *ps[NM];
    auto request = [&]() {
        if (pi >= i1) return;
        if (pkg == 0) {
            const int c = pi / rt_n;
            const size_t t0 = (size_t)(pi - c * rt_n) * kg_n;
            const int e = __ldg(&a.chunks[c * a.chunk_stride]).x;
            pq[0] = (DOWN ? a.L.down_q(e) : a.L.gate_q(e)) + t0 * (NQ * 32);
            ps[0] = (DOWN ? a.L.down_s(e) : a.L.gate_s(e)) + t0 * 8;
            if constexpr (!DOWN) {
                pq[1] = a.L.up_q(e) + t0 * (NQ * 32);
                ps[1] = a.L.up_s(e) + t0 * 8;
            }
        }
        const uint32_t n = (GRP > 1) ? (uint32_t)min(GRP, kg_n - pkg) : 1u;
        if (tc::elect_one()) {
            const uint32_t bar = bar0 + wslot * 8, dst = ring + wslot * S::slot;
            tc::mbar_expect_tx(bar, NM * n * (S::q_bytes + S::s_bytes));
#pragma unroll
            for (int m = 0; m < NM; ++m) {
                tc::bulk_load(dst + m * S::tile, pq[m], n * S::q_bytes, bar);
                if (S::s_bytes) tc::bulk_load(dst + m * S::tile + GRP * S::q_bytes, ps[m], n * S::s_bytes, bar);
            }
        }
        __syncwarp();
#pragma unroll
        for (int m = 0; m < NM; ++m) {
            pq[m] += GRP * NQ * 32;
            ps[m] += GRP * 8;
        }
        if (++wslot == RING) wslot = 0;
        if ((pkg += GRP) >= kg_n) {
            pkg = 0;
            pi += nw;
        }
    };
    if (a.debug_extra_tx != 0 && warp == 0) {
        if (lane == 0) tc::mbar_expect_more(bar0, a.debug_extra_tx);
        __syncwarp();
    }
#pragma unroll 1
    for (int i = 0; i < RING; ++i) request();
    if (DOWN) {
        pdl_wait();
        pdl_trigger();
    }
    const UnpackConst kc = unpack_const_pinned<Q>();
    const int sq_term = xq_term_words(nblk_pad), sq_tok = xq_tok_words(nblk_pad);

    auto item = [&](auto ng_tag, const int4& ch, int rt) {
        constexpr int NG = decltype(ng_tag)::value;
        constexpr int CPG = (TERMS == 1) ? 8 : 4;  // columns of an MMA group
        // This lane's B column of every group (a column past the end repeats the chunk's last one: its sums are not
        // stored). I8: bp = word pairs of the column and term (8 bytes per block), sp = {sx, 8 sx sum q} of the column of
        // the lane's accumulators.
        const uint4* bp[NG];
        const float2* sp[NG];
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            const int n = (TERMS == 1) ? g * CPG + gq : g * CPG + (gq >> 1);
            const int col = ch.y + min(n, ch.z - 1);
            if constexpr (I8) {
                const unsigned* sq = reinterpret_cast<const unsigned*>(a.b);
                bp[g] = reinterpret_cast<const uint4*>(sq + (size_t)col * sq_tok + (gq & 1) * sq_term + t4 * 2);
                sp[g] = reinterpret_cast<const float2*>(sq + (size_t)(ch.y + min(g * CPG + t4, ch.z - 1)) * sq_tok + 2 * sq_term);
            } else {
                const int row = (DOWN || a.col_src_tok == nullptr) ? col : a.col_src_tok[col];
                bp[g] = a.b + ((TERMS == 1) ? (size_t)row : (size_t)row * 2 + (gq & 1)) * a.b_row + t4;
            }
        }
        auto load_b = [&](int g, int b) -> uint4 {  // operand of block b of the group at hand
            if constexpr (I8) {
                const uint2 w = __ldg(reinterpret_cast<const uint2*>(bp[g]) + b * 4);
                const float2 sc = __ldg(sp[g] + b);
                return make_uint4(w.x, w.y, __float_as_uint(sc.x), __float_as_uint(sc.y));
            } else {
                return __ldg(bp[g] + b * 4);
            }
        };
        float acc[NM][NG][4];
#pragma unroll
        for (int m = 0; m < NM; ++m)
#pragma unroll
            for (int g = 0; g < NG; ++g)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[m][g][i] = 0.0f;
        // The next block's activations are loaded one block ahead (at the end of a row that is the first
        // chunk of whatever follows it in the context's memory: loaded, never used), registers permitting.
        constexpr bool AHEAD = NG * NM <= 4;
        uint4 bn[AHEAD ? NG : 1];
        if constexpr (AHEAD) {
#pragma unroll
            for (int g = 0; g < NG; ++g) bn[g] = load_b(g, 0);
        }
        int sub = 0;
#pragma unroll 1
        for (int kg = 0; kg < kg_n; ++kg) {
            if (sub == 0 && !wait_copy(bar0 + rslot * 8, rphase, a.wait_limit_ns)) {
                // The copy has not come within the limit: the lanes raise the status word, wait (with a limit again) for
                // the copies still on their way into this shared memory, and end without storing anything more. They all
                // watch one barrier, whose phase cannot move on before they have passed it, so they come to the same end
                // without a vote; one vote per slot made a 77-token prompt take 2 % longer.
                raise_status(a.status, a.status_host, 4);  // LUMEN_MOE_TIMEOUT
                do {
                    wait_copy(bar0 + rslot * 8, rphase, DRAIN_NS);
                    if (++rslot == RING) {
                        rslot = 0;
                        rphase ^= 1u;
                    }
                } while (rslot != wslot);
                asm volatile("exit;");
                __builtin_unreachable();
            }
            WTile<Q> w[NM];
            const uint32_t src = ring + rslot * S::slot;
#pragma unroll
            for (int m = 0; m < NM; ++m) {
#pragma unroll
                for (int j = 0; j < NQ; ++j) w[m].q[j] = tc::lds128(src + m * S::tile + sub * S::q_bytes + j * 512 + lane * 16);
                if (Q != BF16) w[m].s = tc::lds128(src + m * S::tile + GRP * S::q_bytes + sub * S::s_bytes + gq * 16);
            }
            if (GRP == 1 || ++sub == GRP || kg + 1 == kg_n) {
                sub = 0;
                // every lane's reads of the slot are ordered before the bulk copy that fills it again
                tc::fence_proxy_async();
                __syncwarp();
                if (++rslot == RING) {
                    rslot = 0;
                    rphase ^= 1u;
                }
                request();
            }
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                uint4 bc[NG];
#pragma unroll
                for (int g = 0; g < NG; ++g) {
                    if constexpr (AHEAD) {
                        bc[g] = bn[g];
                        bn[g] = load_b(g, b + 1);
                    } else {
                        bc[g] = load_b(g, b);
                    }
                }
#pragma unroll
                for (int m = 0; m < NM; ++m) {
                    const float2 sc = block_scales<Q>(w[m], b);
                    if constexpr (I8) {
                        const uint4 qv = w[m].q[(b >> 1) % NQ];
                        const unsigned w0 = (b & 1) ? qv.z : qv.x, w8 = (b & 1) ? qv.w : qv.y;
#pragma unroll
                        for (int g = 0; g < NG; ++g) {
                            int c[4] = {0, 0, 0, 0};
                            mma_u8s8(c, w0 & 0x0F0F0F0Fu, w8 & 0x0F0F0F0Fu, (w0 >> 4) & 0x0F0F0F0Fu, (w8 >> 4) & 0x0F0F0F0Fu,
                                     bc[g].x, bc[g].y);
                            const float sx = __uint_as_float(bc[g].z), off = __uint_as_float(bc[g].w), k1 = 1.0f / 254.0f;
                            acc[m][g][0] = fmaf(sc.x, fmaf(sx, fmaf((float)c[1], k1, (float)c[0]), -off), acc[m][g][0]);
                            acc[m][g][2] = fmaf(sc.y, fmaf(sx, fmaf((float)c[3], k1, (float)c[2]), -off), acc[m][g][2]);
                        }
                    } else {
                        uint32_t lo[4], hi[4];
                        unpack_block<Q>(w[m], b, lo, hi, kc);
#pragma unroll
                        for (int g = 0; g < NG; ++g) block_mma<Q, TERMS>(lo, hi, sc, bc[g], acc[m][g]);
                    }
                }
            }
#pragma unroll
            for (int g = 0; g < NG; ++g) {
                bp[g] += I8 ? 8 : 16;  // one group on: 4 blocks x 32 | 64 bytes
                if (I8) sp[g] += 4;
            }
        }
        // lane: rows gq and gq + 8 of the tile, MMA columns 2 t4, 2 t4 + 1 of each group
        const int r0 = rt * 16 + gq;
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            if constexpr (MODE == DOWN_1) {
                // transposed through the tensor path's 8 x 8 move, so that a lane holds two neighbouring rows of one
                // column: four lanes then write 16 bytes of an output row
                const uint32_t p0 = movmatrix_trans(h2_bits(acc[0][g][0], acc[0][g][1]));
                const uint32_t p1 = movmatrix_trans(h2_bits(acc[0][g][2], acc[0][g][3]));
                const int n = g * 8 + gq;
                if (n < ch.z) {
                    int orow = ch.y + n;
                    if (a.out_row_map) orow = a.out_row_map[orow];
                    __half* dst = a.out16;
                    bool live = true;
                    if (a.peer.ret_map != nullptr) {
                        // plain stores into the return buffer of the rank the row came from
                        const int m = a.peer.ret_map[orow];
                        const int pr = (m >> 24) & 0xff;
                        orow = m & 0xffffff;
                        live = pr < a.peer.world && orow < a.peer.rows_cap;  // never leave the buffers
                        if (live) dst = a.peer.base[pr];
                    }
                    if (live) {
                        uint32_t* d = reinterpret_cast<uint32_t*>(dst + (size_t)orow * a.L.H + rt * 16 + 2 * t4);
                        d[0] = p0;
                        d[4] = p1;
                    }
                }
            } else if constexpr (MODE == GATE_UP_1) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int n = g * 8 + 2 * t4 + (i & 1), row = r0 + (i >> 1) * 8;
                    if (n < ch.z) {
                        // fast exp and divide: their error (~2^-21) is far below the f16 rounding that follows
                        const float gt = acc[0][g][i];
                        a.out16[(size_t)(ch.y + n) * a.L.I + (row & ~31) + perm32(row & 31)] =
                            __float2half_rn(__fdividef(gt, 1.0f + __expf(-gt)) * acc[NM - 1][g][i]);
                    }
                }
            } else {
                const int n = g * 4 + t4;
                if (n < ch.z) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float v = acc[0][g][2 * i] + acc[0][g][2 * i + 1];
                        if constexpr (DOWN) {
                            __stcg(a.d32 + (size_t)(ch.y + n) * a.L.H + r0 + i * 8, v);
                        } else {
                            const float up = acc[NM - 1][g][2 * i] + acc[NM - 1][g][2 * i + 1];
                            store_swiglu_frag<Q>(a.sf, ch.y + n, r0 + i * 8, a.L.kg_i * 4, (v / (1.0f + expf(-v))) * up);
                        }
                    }
                }
            }
        }
    };
    for (int i = i0 + warp; i < i1; i += nw) {
        const int c = i / rt_n;
        const int4 ch = __ldg(&a.chunks[c * a.chunk_stride]);
        const int rt = i - c * rt_n;
        const int ng = (TERMS == 1) ? (ch.z + 7) >> 3 : (ch.z + 3) >> 2;
        if (ng == 1) item(std::integral_constant<int, 1>{}, ch, rt);
        else if (ng == 2) item(std::integral_constant<int, 2>{}, ch, rt);
        else item(std::integral_constant<int, 4>{}, ch, rt);
    }
}

// out[t] = residual[t] + sum_slot w * d32[column of the slot], in slot order (cuda/shaders/moe_accum.cu:22-46). Two outputs
// a thread. PAIRS: residual and out, the caller's rows of f32, lie on 8-byte boundaries; else they are read and written
// one by one (d32 is the context's own and always aligned).
template <bool PAIRS>
__global__ void __launch_bounds__(128)
combine_f32_kernel(const float* __restrict__ d32, RouteDev R, const float* residual, float* out, int H, int K) {
    const int t = blockIdx.x, h = (blockIdx.y * 128 + threadIdx.x) * 2;
    // (the tables are the router's, complete before the down kernel started)
    int col[MAX_TOP_K];
    float w[MAX_TOP_K];
#pragma unroll
    for (int s = 0; s < MAX_TOP_K; ++s)
        if (s < K) {
            col[s] = __ldg(R.dst_to_col + t * K + s);
            w[s] = __ldg(R.weights + t * K + s);
        }
    pdl_trigger();
    pdl_wait();
    if (h >= H) return;
    const float* res = residual + (size_t)t * H + h;
    float2 acc = PAIRS ? *reinterpret_cast<const float2*>(res) : make_float2(res[0], res[1]);
    float2 d[MAX_TOP_K];
#pragma unroll
    for (int s = 0; s < MAX_TOP_K; ++s)
        if (s < K) d[s] = __ldcg(reinterpret_cast<const float2*>(d32 + (size_t)col[s] * H + h));
#pragma unroll
    for (int s = 0; s < MAX_TOP_K; ++s)
        if (s < K) {
            acc.x = __fadd_rn(acc.x, __fmul_rn(w[s], d[s].x));
            acc.y = __fadd_rn(acc.y, __fmul_rn(w[s], d[s].y));
        }
    float* dst = out + (size_t)t * H + h;
    if (PAIRS) {
        *reinterpret_cast<float2*>(dst) = acc;
    } else {
        dst[0] = acc.x;
        dst[1] = acc.y;
    }
}

// chained: the kernel in front in the stream waits for the routing kernels before it lets this one start (see above)
template <int Q, int MODE, int WARPS = default_warps<Q, MODE>()>
cudaError_t launch_t(const Args& a, int sms, cudaStream_t st, bool chained = true) {
    auto* kern = stream_kernel<Q, MODE, WARPS>;
    constexpr size_t smem = Shape<Q, MODE, WARPS>::smem;
    static SmemOptIn optin;
    const cudaError_t e = ensure_dyn_smem(kern, smem, optin);
    if (e != cudaSuccess) return e;
    count_launch();
    if (!chained) {
        kern<<<sms, WARPS * 32, smem, st>>>(a);
        return cudaGetLastError();
    }
    return launch_dep(kern, dim3(sms), dim3(WARPS * 32), smem, st, a);
}

template <int MODE>
cudaError_t launch_q(const Args& a, int sms, cudaStream_t st, bool chained = true) {
    switch (a.L.quant) {
        case Q4_0: return launch_t<Q4_0, MODE>(a, sms, st, chained);
        case Q8_0: return launch_t<Q8_0, MODE>(a, sms, st, chained);
        default:
            if constexpr (MODE == GATE_UP_1 || MODE == DOWN_1) return cudaErrorInvalidValue;  // (prefill_streams takes none)
            else return launch_t<BF16, MODE>(a, sms, st, chained);
    }
}

static uint32_t limit_ns(unsigned wait_limit_us) { return wait_limit_us ? wait_limit_us * 1000u : (uint32_t)tc::WAIT_LIMIT_NS; }

// decode batches: the router's work records are the chunks (an expert has at most sixteen columns)
static Args decode_args(const DecodeArgs& p) {
    Args g{};
    g.status = p.status;
    g.status_host = p.status_host;
    g.wait_limit_ns = limit_ns(p.wait_limit_us);
    g.L = p.L;
    g.chunks = p.R.work;
    g.chunk_stride = 2;
    g.n_chunks = p.R.n_uexp;
    return g;
}

// Items of an SM in a decode batch: rt rows of tiles of every expert that the tokens' choices hit, as many as under near-uniform routing.
// margin: so many more, for a choice that loses where the tokens hit more experts than that.
static int items_per_sm(const DecodeArgs& p, int rt, float margin = 0.0f) {
    float miss = 1.0f;
    for (int t = 0; t < p.T; ++t) miss *= 1.0f - (float)p.K / (float)p.L.E;
    return (int)ceilf((float)p.L.E * (1.0f - miss) * (float)rt / (float)p.sms + margin);
}
static int rounds(int items, int warps) { return (items + warps - 1) / warps; }

}  // namespace stream

// gate/up of a decode batch: hi + lo activation fragments by token, SwiGLU fragments for the down product
cudaError_t launch_stream_gate_up(const DecodeArgs& p, cudaStream_t st) {
    stream::Args g = stream::decode_args(p);
    g.col_src_tok = p.R.col_src_tok;
    g.b = p.xf;
    g.b_row = (size_t)p.L.kg_h * 16;
    g.sf = p.sf;
    g.debug_extra_tx = p.debug_expire;
    // BF16: ten warps where they take a round less than eight, up to two rounds (eight and ten, us replayed, by items an SM. H = 2048, I = 768, E = 128: 10
    // 65.2 and 60.2, 12 70.7 and 72.9, 14 79.2 and 80.4, 17 98.5 and 94.6, 23 119.9 and 122.6, 25 137.2 and 136.1; I = 512, E = 256: 7 48.7
    // and 48.7, 9 63.1 and 56.6, 13 80.5 and 81.5, 18 105.8 and 103.5; H = 3072, I = 1024, E = 32: 10 93 and 80; H = 4096, I = 1536, E = 64: 11 123.7
    // and 126.5, 14 146 and 150, 19 184 and 178, 31 295 and 303. Three rounds for four gain 2 % at most, as 25 above, and one call loses by them: H = 4096, I = 1536,
    // E = 64: 24.4 222 and 242)
    const int n = stream::items_per_sm(p, p.L.rt_i);
    if (p.L.quant == BF16 && n <= 20 && stream::rounds(n, 10) < stream::rounds(n, 8)) return stream::launch_t<BF16, stream::GATE_UP_2, 10>(g, p.sms, st);
    return stream::launch_q<stream::GATE_UP_2>(g, p.sms, st);
}

// down + combine of a decode batch; int8: the SwiGLU outputs are in p.sq (Q4_0), else fragments in p.sf. after_gate_up: the
// gate/up kernel is in front of it in the stream
cudaError_t launch_stream_down(const DecodeArgs& p, bool int8, bool after_gate_up, cudaStream_t st) {
    stream::Args d = stream::decode_args(p);
    d.b = int8 ? reinterpret_cast<const uint4*>(p.sq) : p.sf;
    d.b_row = (size_t)p.L.kg_i * 16;
    d.d32 = p.d32;
    d.debug_extra_tx = int8 ? p.debug_expire : 0;  // (the chain's first streaming kernel)
    // More warps where they take a round less. Q8_0, whose rings get shorter for it: up to two rounds (16 and 20 warps, us replayed, by items an SM.
    // H = 2048, I = 768, E = 128: 20 40.2 and 38.9, 26 44.1 and 44.8, 31 47.7 and 48.2, 36 53.5 and 51.6, 45 71.4 and 72.5, 60 85.1 and 85.9;
    // H = 2048, I = 1408, E = 64: 19 53.4 and 50.4, 23 63.5 and 65.7, 27 74 and 75.5; H = 3072, I = 1024, E = 32: 18 45.1 and 43.6, 23 49.7
    // and 51.6, 34 71.4 and 69.5), with half an item to spare: at the brink the tokens often hit an expert more, and a round more it is (H = 2048,
    // I = 1408, E = 64: 40.0 105.7 and 114.0; H = 4096, I = 1536, E = 64: 19.8 62.3 and 65.9; H = 4096, I = 512, E = 64: 19.54 46.3 and 47.6).
    // BF16: any number, while the batch's fragments are not too many (8 and 12 warps. H = 2048, I = 768, E = 128: 14 39.0 and 39.0, 36 79.2 and 77.2;
    // H = 1024, I = 384, E = 64: 8 21.8 and 22.2, 9 24.1 and 23.1, 15 29.1 and 29.4; 256 KB: 16 tokens of I = 512
    // 125.0 and 124.5, of H = 3072, I = 1024, E = 32 113 and 111; beyond: H = 4096, I = 1536, E = 64 8 tokens, 288 KB, 211 and 215, 16 tokens 295 and 322).
    const int n = stream::items_per_sm(p, p.L.rt_h);
    const int spare = stream::items_per_sm(p, p.L.rt_h, 0.5f);
    const bool more = p.L.quant == BF16 ? (size_t)p.T * p.K * p.L.kg_i * 512 <= 256 * 1024 && stream::rounds(n, 12) < stream::rounds(n, 8)
                                        : spare <= 40 && stream::rounds(spare, 20) < stream::rounds(n, 16);
    // Q4_0: 20 warps from 10 items an SM on. Fewer are one round of 16 warps with room for their longer rings (16 and 20 warps, us replayed, by items an
    // SM: a lone expert of 1024 x 2816, 0.4, 11 tokens 35.9 and 40.3; 1024 x 2816, E = 8, 3.4 41.1 and 46.5; 1024 x 512, E = 32, 11.7 20.3 and 19.7; 1024 x
    // 768, E = 128, 17.8 27.6 and 25.9; 2048 x 1408, E = 64, 21.5 39.8 and 35.2, 38 59.1 and 55.2; 2048 x 768, E = 128, 25 29.4 and 30.1, 35.5 37.2 and 35.1,
    // 71 61.5 and 60.6; the worst 4096 x 512, E = 64, 25 40.6 and 41.7)
    const cudaError_t e = int8 && n > 10                   ? stream::launch_t<Q4_0, stream::DOWN_2I, 20>(d, p.sms, st, after_gate_up)
                          : int8                           ? stream::launch_t<Q4_0, stream::DOWN_2I>(d, p.sms, st, after_gate_up)
                          : more && p.L.quant == BF16      ? stream::launch_t<BF16, stream::DOWN_2, 12>(d, p.sms, st, after_gate_up)
                          : more && p.L.quant == Q8_0      ? stream::launch_t<Q8_0, stream::DOWN_2, 20>(d, p.sms, st, after_gate_up)
                                                           : stream::launch_q<stream::DOWN_2>(d, p.sms, st, after_gate_up);
    if (e != cudaSuccess) return e;
    count_launch();
    // (H is a multiple of 32, so every row lies on the boundary that the first one does)
    const bool pairs = (reinterpret_cast<uintptr_t>(p.residual) | reinterpret_cast<uintptr_t>(p.out)) % 8 == 0;
    return launch_dep(pairs ? stream::combine_f32_kernel<true> : stream::combine_f32_kernel<false>, dim3(p.T, (p.L.H / 2 + 127) / 128), dim3(128), 0, st, (const float*)p.d32, p.R,
                      p.residual, p.out, p.L.H, p.K);
}

// Expert products of a short prompt: x16 rows by token (planes' element order), s16 by column.
cudaError_t launch_stream_prefill(const PrefillArgs& p, const __half* x16, __half* out16_rows, cudaStream_t st,
                                  const TcPeerOut* peer) {
    stream::Args g{};
    g.L = p.L;
    g.chunks = p.tiles;
    g.chunk_stride = 1;
    g.n_chunks = p.n_tiles;
    g.starts = p.stream_starts;
    g.col_src_tok = p.R.col_src_tok;
    g.b = reinterpret_cast<const uint4*>(x16);
    g.b_row = (size_t)p.L.H / 8;
    g.out16 = p.s16;
    g.status = p.status;
    g.status_host = p.status_host;
    g.wait_limit_ns = stream::limit_ns(p.wait_limit_us);
    g.debug_extra_tx = p.debug_extra_tx;
    const cudaError_t e = stream::launch_q<stream::GATE_UP_1>(g, p.sms, st);
    if (e != cudaSuccess) return e;
    stream::Args d = g;
    d.debug_extra_tx = 0;  // the hook applies to the first kernel of the pair
    d.starts = p.stream_starts ? p.stream_starts + p.sms + 1 : nullptr;
    d.b = reinterpret_cast<const uint4*>(p.s16);
    d.b_row = (size_t)p.L.I / 8;
    d.out16 = out16_rows ? out16_rows : p.d16;
    d.out_row_map = out16_rows ? p.R.col_src_tok : nullptr;
    if (peer) d.peer = *peer;
    // (24 warps of Q4_0, with the 80 registers that they leave, gain up to 4 % under even loads and lose 6-14 % where some experts have several
    // operands of eight columns, which the host cannot see: 83 tokens of 2048 x 768, E = 128, 121 and 117 us, with Zipf loads 144 and
    // 158; 64 tokens of 4096 x 1536, E = 64, 222 and 212, 280 and 299)
    return stream::launch_q<stream::DOWN_1>(d, p.sms, st);
}

}  // namespace lumen
