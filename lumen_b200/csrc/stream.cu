// Expert products for batches in which an expert has few columns (decode batches, short prompts):
// weights streamed once, multiplied on the warp-level tensor cores straight from registers.
//
// With a handful of columns per expert a layer call reads every selected expert's weights (340 MB
// at H=2048, I=768, E=128, Q4_0) for little arithmetic. The tcgen05 kernel (prefill_tc.cu) has
// to write each dequantised weight to shared memory as a rounded f16 operand: ~350 instructions per
// 16 x 128 tile, which is what bounds it there (60 % issue slots, 1.9 TB/s at 77 tokens). Here a
// weight goes from the quant planes to an mma.sync fragment as an exact small integer, the f32 scale is
// applied to the block's sums, and nothing is written back: ~110 instructions per tile at up to
// eight columns, ~30 more per further eight.
//
// A WARP owns an item (16 output rows of one expert times one chunk of its columns, all inputs). Items are
// dealt to the CTAs (one per SM) as equal contiguous ranges, so that the warps of an SM work on neighbouring
// rows of one expert and share its activations in L1; inside the range the warps take every
// WARPS-th item. Each warp keeps a ring of 128-input groups in flight with bulk copies on its own
// mbarriers, across item boundaries: no CTA-wide synchronisation anywhere in the loop.
//
//   gate_up   16 rows of I: gate and up tiles together, SwiGLU at the end
//             (cuda/shaders/moe_expert_q4_0.cu:58-108, moe_expert.cu:47-97)
//   down      16 rows of H (moe_grouped.cu:1202-1510); the weighted sum follows in scatter_accum_kernel
//
// TERMS = 1 (prompts): activations are single f16 rows in the planes' element order (x16, s16), the
// precision of the tcgen05 path. TERMS = 2 (decode): hi + lo fragments, two MMA columns per token.
// Every wait is bounded; a warp whose wait runs out raises the context's status word.
#include "decode_common.cuh"
#include "tc_common.cuh"
#include <type_traits>

namespace lumen {

namespace stream {

using namespace dcommon;

template <int Q>
struct Cfg;  // a ring slot holds up to GRP 128-input groups (of each matrix); RING_GU / RING_DN slots per warp
// (the copy peak times the latency is ~55 KB per SM in flight; the rings hold 139..184 KB)
template <>
struct Cfg<Q4_0> {
    static constexpr int WARPS = 16, GRP = 2, RING_GU = 2, RING_DN = 4;
};
template <>
struct Cfg<Q8_0> {
    static constexpr int WARPS = 16, GRP = 1, RING_GU = 2, RING_DN = 4;
};
template <>
struct Cfg<BF16> {
    static constexpr int WARPS = 8, GRP = 1, RING_GU = 2, RING_DN = 4;
};

template <int Q>
struct Raw {  // one 16-row x 128-input tile: quants then scales
    static constexpr int q_bytes = QTraits<Q>::NQ * 512, s_bytes = (Q == BF16) ? 0 : 128, bytes = q_bytes + s_bytes;
};

struct Args {
    LayerDev L;
    const int4* chunks;         // {expert, first column, columns, -}
    const int32_t* starts;      // [CTAs + 1] first item of every CTA (null: equal shares of n_chunks)
    const int32_t* n_chunks;
    const int32_t* col_src_tok;
    const uint4* b;             // activation rows: TERMS 1: f16 [row][kdim]; TERMS 2: fragments [row][2][nblk_pad][4]
    size_t b_row;               // uint4 per row (TERMS 2: per row and term)
    __half* out16;              // TERMS 1: s16 [C, I] (permuted order) | d16 [C, H]
    uint4* sf;                  // TERMS 2 gate/up: SwiGLU fragments
    int32_t* status;
    int32_t* status_host;
    uint64_t wait_limit_ns;
    int debug_extra_tx;             // test hook: every warp's first group expects this many bytes too many
    const int32_t* out_row_map;     // down: output row of compact column c (null = c itself)
    TcPeerOut peer;                 // down, expert parallel: output rows go to other ranks' buffers (ret_map null = off)
};

// b fragments of the block's two MMAs out of one 16-byte chunk (the two layouts order them differently)
template <int TERMS>
__device__ __forceinline__ void b_regs(const uint4& v, uint32_t& l0, uint32_t& l1, uint32_t& h0, uint32_t& h1) {
    l0 = v.x;
    l1 = (TERMS == 1) ? v.z : v.y;
    h0 = (TERMS == 1) ? v.y : v.z;
    h1 = v.w;
}

// A bf16 pair as an f16 pair (exact for normal f16 magnitudes, as the f16 copies of the tcgen05 path)
__device__ __forceinline__ uint32_t bf2_to_h2(uint32_t v) {
    const __half2 h = __floats2half2_rn(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
    return *reinterpret_cast<const uint32_t*>(&h);
}

template <int Q, int TERMS>
__device__ __forceinline__ void unpack(const WTile<Q>& w, int b, uint32_t (&lo)[4], uint32_t (&hi)[4], const UnpackConst& k) {
    unpack_block<Q>(w, b, lo, hi, k);
    if (Q == BF16 && TERMS == 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            lo[i] = bf2_to_h2(lo[i]);
            hi[i] = bf2_to_h2(hi[i]);
        }
    }
}

// acc += scale * (block b of the tile) x (eight columns)
template <int Q, int TERMS>
__device__ __forceinline__ void block_mma(const uint32_t (&lo)[4], const uint32_t (&hi)[4], const float2 sc, const uint4& bv,
                                          float (&acc)[4]) {
    uint32_t l0, l1, h0, h1;
    b_regs<TERMS>(bv, l0, l1, h0, h1);
    if constexpr (Q == BF16) {
        if constexpr (TERMS == 1) {
            mma_f16(acc, lo, l0, l1);
            mma_f16(acc, hi, h0, h1);
        } else {
            mma_bf16(acc, lo, l0, l1);
            mma_bf16(acc, hi, h0, h1);
        }
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

template <int Q, int TERMS, bool DOWN>
__global__ void __launch_bounds__(Cfg<Q>::WARPS * 32, 1)
stream_kernel(const __grid_constant__ Args a) {
    static_assert(!DOWN || TERMS == 1, "the decode chain has its own down kernel");
    constexpr int WARPS = Cfg<Q>::WARPS, RING = DOWN ? Cfg<Q>::RING_DN : Cfg<Q>::RING_GU;
    constexpr int NM = DOWN ? 1 : 2;  // matrices of an item: down | gate and up
    constexpr int GRP = Cfg<Q>::GRP;
    constexpr uint32_t RAW_Q = Raw<Q>::q_bytes, RAW_S = Raw<Q>::s_bytes, RAW = GRP * (RAW_Q + RAW_S), SLOT = NM * RAW;
    extern __shared__ __align__(128) uint8_t ring_smem[];  // [WARPS][RING][NM][quants of GRP groups | scales of GRP groups]
    __shared__ uint64_t bar_s[WARPS * RING];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gq = lane >> 2, t4 = lane & 3;
    const uint32_t ring0 = tc::smem_u32(ring_smem) + (uint32_t)warp * RING * SLOT;
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
    int i0, i1;
    if (a.starts != nullptr) {
        i0 = a.starts[blockIdx.x];
        i1 = a.starts[blockIdx.x + 1];
    } else {
        const int total = *a.n_chunks * rt_n;
        i0 = (int)((long long)total * blockIdx.x / gridDim.x);
        i1 = (int)((long long)total * (blockIdx.x + 1) / gridDim.x);
    }

    // request cursor: next group (item pi, group pkg) to copy
    int pi = i0 + warp, pkg = 0, issued = 0, taken = 0;
    const uint4 *pq[NM], *ps[NM];
    auto top_up = [&]() {
        while (issued - taken < RING && pi < i1) {
            if (pkg == 0) {
                const int c = pi / rt_n;
                const size_t t0 = (size_t)(pi - c * rt_n) * kg_n;
                const int e = __ldg(&a.chunks[c]).x;
                pq[0] = (DOWN ? a.L.down_q(e) : a.L.gate_q(e)) + t0 * (RAW_Q / 16);
                ps[0] = (DOWN ? a.L.down_s(e) : a.L.gate_s(e)) + t0 * 8;
                if constexpr (!DOWN) {
                    pq[1] = a.L.up_q(e) + t0 * (RAW_Q / 16);
                    ps[1] = a.L.up_s(e) + t0 * 8;
                }
            }
            const int slot = issued % RING;
            const uint32_t n = (GRP > 1) ? (uint32_t)min(GRP, kg_n - pkg) : 1u;
            if (lane == 0) {
                const uint32_t bar = bar0 + slot * 8, dst = ring0 + slot * SLOT;
                tc::mbar_expect_tx(bar, NM * n * (RAW_Q + RAW_S) + (issued == 0 ? (uint32_t)a.debug_extra_tx : 0u));
#pragma unroll
                for (int m = 0; m < NM; ++m) {
                    tc::bulk_load(dst + m * RAW, pq[m], n * RAW_Q, bar);
                    if (RAW_S) tc::bulk_load(dst + m * RAW + GRP * RAW_Q, ps[m], n * RAW_S, bar);
                }
            }
#pragma unroll
            for (int m = 0; m < NM; ++m) {
                pq[m] += GRP * RAW_Q / 16;
                ps[m] += GRP * 8;
            }
            ++issued;
            if ((pkg += GRP) >= kg_n) {
                pkg = 0;
                pi += WARPS;
            }
        }
    };
    top_up();
    if (DOWN) {
        pdl_wait();
        pdl_trigger();
    }
    bool ok = true;
    auto wait_slot = [&]() -> bool {
        const uint32_t bar = bar0 + (taken % RING) * 8, ph = (taken / RING) & 1;
        bool r = tc::mbar_try(bar, ph);
        if (!r) {
            const uint64_t t0 = tc::globaltimer_ns();
            do {
                r = tc::mbar_try(bar, ph);
            } while (!r && tc::globaltimer_ns() - t0 < a.wait_limit_ns);
        }
        return __all_sync(0xffffffffu, r);
    };

    const UnpackConst kc = unpack_const_pinned<Q>();
    auto item = [&](auto ng_tag, const int4& ch, int rt) {
        constexpr int NG = decltype(ng_tag)::value;
        constexpr int CPG = (TERMS == 1) ? 8 : 4;  // columns of an MMA group
        const uint4* bp[NG];
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            // this lane's B column; a column past the end repeats the chunk's last one (its sums are not stored)
            const int n = (TERMS == 1) ? g * CPG + gq : g * CPG + (gq >> 1);
            const int col = ch.y + min(n, ch.z - 1);
            const int row = (DOWN || a.col_src_tok == nullptr) ? col : a.col_src_tok[col];
            bp[g] = a.b + ((TERMS == 1) ? (size_t)row : (size_t)row * 2 + (gq & 1)) * a.b_row + t4;
        }
        float acc[NM][NG][4];
#pragma unroll
        for (int m = 0; m < NM; ++m)
#pragma unroll
            for (int g = 0; g < NG; ++g)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[m][g][i] = 0.0f;
        // The next block's activations are loaded one block ahead (at the end of a row that is the first
        // chunk of whatever follows it in the context's memory: loaded, never used).
        uint4 bn[NG];
#pragma unroll
        for (int g = 0; g < NG; ++g) bn[g] = __ldg(bp[g]);
        int sub = GRP;  // next group within the slot
        uint32_t src = 0;
#pragma unroll 1
        for (int kg = 0; kg < kg_n; ++kg) {
            if (GRP == 1 || sub == GRP) {
                ok = wait_slot();
                if (!ok) return;
                src = ring0 + (taken % RING) * SLOT;
                sub = 0;
            }
            WTile<Q> w[NM];
#pragma unroll
            for (int m = 0; m < NM; ++m) {
#pragma unroll
                for (int j = 0; j < QTraits<Q>::NQ; ++j) w[m].q[j] = tc::lds128(src + m * RAW + sub * RAW_Q + j * 512 + lane * 16);
                if (Q != BF16) w[m].s = tc::lds128(src + m * RAW + GRP * RAW_Q + sub * RAW_S + gq * 16);
            }
            if (GRP == 1 || ++sub == GRP || kg + 1 == kg_n) {
                // every lane's reads of the slot are ordered before the bulk copy that fills it again
                tc::fence_proxy_async();
                __syncwarp();
                ++taken;
                top_up();
            }
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                uint4 bc[NG];
#pragma unroll
                for (int g = 0; g < NG; ++g) {
                    bc[g] = bn[g];
                    bn[g] = __ldg(bp[g] + (b + 1) * 4);
                }
#pragma unroll
                for (int m = 0; m < NM; ++m) {
                    uint32_t lo[4], hi[4];
                    unpack<Q, TERMS>(w[m], b, lo, hi, kc);
                    const float2 sc = block_scales<Q>(w[m], b);
#pragma unroll
                    for (int g = 0; g < NG; ++g) block_mma<Q, TERMS>(lo, hi, sc, bc[g], acc[m][g]);
                }
            }
#pragma unroll
            for (int g = 0; g < NG; ++g) bp[g] += 16;
        }
        // lane: rows gq and gq + 8 of the tile, MMA columns 2 t4, 2 t4 + 1 of each group
        const int r0 = rt * 16 + gq;
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            if constexpr (DOWN) {
                // transposed through the tensor path's 8 x 8 move, so that a lane holds two neighbouring rows of one
                // column: four lanes then write 16 bytes of an output row
                uint32_t p0 = h2_bits(acc[0][g][0], acc[0][g][1]), p1 = h2_bits(acc[0][g][2], acc[0][g][3]);
                p0 = movmatrix_trans(p0);
                p1 = movmatrix_trans(p1);
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
            } else if constexpr (TERMS == 1) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int n = g * 8 + 2 * t4 + (i & 1), row = r0 + (i >> 1) * 8;
                    if (n < ch.z) {
                        {
                            // fast exp and divide: their error (~2^-21) is far below the f16 rounding that follows
                            const float gt = acc[0][g][i];
                            a.out16[(size_t)(ch.y + n) * a.L.I + (row & ~31) + perm32(row & 31)] =
                                __float2half_rn(__fdividef(gt, 1.0f + __expf(-gt)) * acc[NM - 1][g][i]);
                        }
                    }
                }
            } else {
                const int n = g * 4 + t4;
                if (n < ch.z) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float gt = acc[0][g][2 * i] + acc[0][g][2 * i + 1];
                        const float up = acc[NM - 1][g][2 * i] + acc[NM - 1][g][2 * i + 1];
                        store_swiglu_frag<Q>(a.sf, ch.y + n, r0 + i * 8, a.L.kg_i * 4, (gt / (1.0f + expf(-gt))) * up);
                    }
                }
            }
        }
    };
    for (int i = i0 + warp; i < i1 && ok; i += WARPS) {
        const int c = i / rt_n;
        const int4 ch = __ldg(&a.chunks[c]);
        const int rt = i - c * rt_n;
        const int ng = (TERMS == 1) ? (ch.z + 7) >> 3 : (ch.z + 3) >> 2;
        if (ng == 1) item(std::integral_constant<int, 1>{}, ch, rt);
        else if (ng == 2) item(std::integral_constant<int, 2>{}, ch, rt);
        else if (ng == 3) item(std::integral_constant<int, 3>{}, ch, rt);
        else item(std::integral_constant<int, 4>{}, ch, rt);
    }
    if (!ok) {
        // give-up: let the copies in flight land before the shared memory goes away
        for (; taken != issued; ++taken)
            for (int k = 0; k < (1 << 16) && !tc::mbar_try(bar0 + (taken % RING) * 8, (taken / RING) & 1); ++k) {}
        if (lane == 0) raise_status(a.status, a.status_host, 4);  // LUMEN_MOE_TIMEOUT
    }
}

template <int Q, int TERMS, bool DOWN>
cudaError_t launch_t(const Args& a, int sms, cudaStream_t st) {
    constexpr size_t smem = (size_t)Cfg<Q>::WARPS * (DOWN ? Cfg<Q>::RING_DN : Cfg<Q>::RING_GU) * (DOWN ? 1 : 2) * Cfg<Q>::GRP * Raw<Q>::bytes;
    static SmemOptIn optin;
    const cudaError_t e = ensure_dyn_smem(stream_kernel<Q, TERMS, DOWN>, smem, optin);
    if (e != cudaSuccess) return e;
    count_launch();
    return launch_dep(stream_kernel<Q, TERMS, DOWN>, dim3(sms), dim3(Cfg<Q>::WARPS * 32), smem, st, a);
}

template <int TERMS, bool DOWN>
cudaError_t launch_q(const Args& a, int sms, cudaStream_t st) {
    switch (a.L.quant) {
        case Q4_0: return launch_t<Q4_0, TERMS, DOWN>(a, sms, st);
        case Q8_0: return launch_t<Q8_0, TERMS, DOWN>(a, sms, st);
        default: return launch_t<BF16, TERMS, DOWN>(a, sms, st);
    }
}

}  // namespace stream

// Activation rows of a prompt for both products: x16 rows by token (planes' element order), s16 by column.
cudaError_t launch_stream_prefill(const PrefillArgs& p, const __half* x16, __half* out16_rows, cudaStream_t st,
                                  const TcPeerOut* peer) {
    stream::Args g{};
    g.L = p.L;
    g.chunks = p.tiles;
    g.n_chunks = p.n_tiles;
    g.starts = p.stream_starts;
    g.col_src_tok = p.R.col_src_tok;
    g.b = reinterpret_cast<const uint4*>(x16);
    g.b_row = (size_t)p.L.H / 8;
    g.out16 = p.s16;
    g.status = p.status;
    g.status_host = p.status_host;
    g.wait_limit_ns = p.wait_limit_us ? (uint64_t)p.wait_limit_us * 1000ull : tc::WAIT_LIMIT_NS;
    g.debug_extra_tx = p.debug_extra_tx;
    cudaError_t e = stream::launch_q<1, false>(g, p.sms, st);
    if (e != cudaSuccess) return e;
    stream::Args d = g;
    d.debug_extra_tx = 0;  // the hook applies to the first kernel of the pair
    d.starts = p.stream_starts ? p.stream_starts + p.sms + 1 : nullptr;
    d.b = reinterpret_cast<const uint4*>(p.s16);
    d.b_row = (size_t)p.L.I / 8;
    d.out16 = out16_rows ? out16_rows : p.d16;
    if (peer) d.peer = *peer;
    d.out_row_map = out16_rows ? p.R.col_src_tok : nullptr;
    return stream::launch_q<1, true>(d, p.sms, st);
}

}  // namespace lumen
