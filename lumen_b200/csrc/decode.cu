// Decode path (1..16 tokens) of the MoE FFN as a chain of kernels launched as programmatic dependents: the
// router here, the expert products in decode_small.cu and stream.cu; the rule between chain and fused kernel; and
// the gate/up and down kernels of the mma.sync prefill path.
//
//   router_small_kernel   one or two expert rows per CTA: router logit(s) W_r[e]·x[t]
//                         (moe_router_logits_v2, cuda/shaders/moe_batched.cu:708),
//                         optional fused FFN RMSNorm (cuda/shaders/norm.cu:28-76),
//                         activation fragments; the last CTA to finish (fence +
//                         ticket, no spinning) does gating/top-k/renorm
//                         (cuda/moe.rs:6464-6504) and the stable counting sort
//                         (cuda/moe.rs:2115-2147).
//   gate_up_kernel        per (distinct expert, 16 rows of I): gate and up rows
//                         times the tokens routed to the expert, SwiGLU
//                         (cuda/shaders/moe_expert_q4_0.cu:58-108, moe_expert.cu:62-97).
//                         The form of the mma.sync prefill path; decode batches take
//                         gate_up_stream_kernel (decode_small.cu) or the kernel of stream.cu.
//   down_general_kernel   its down product (moe_expert_q4_0.cu:118-151).
//
// The products are HBM-bound: each weight byte is read once with 128-bit loads, and the
// arithmetic runs on the tensor cores (mma_frag.cuh).
#include "decode_common.cuh"
#include <type_traits>
#include "router.cuh"

namespace lumen {

using dcommon::pdl_trigger;
using dcommon::pdl_wait;

constexpr int RS_THREADS = 512;  // 16 warps: the last CTA gates one token per warp at batches up to 16
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_BLOCKS = RS_THREADS / 8;  // 32-input blocks of the activation operand an operand CTA builds

// Sums v[0..15] over the warp's lanes in 16 shuffles instead of 80: every step halves the values a lane
// is responsible for. Returns the total of value lane >> 1.
__device__ __forceinline__ float warp_sum16(float (&v)[16]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16, n = 8; n >= 1; o >>= 1, n >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float keep = up ? v[i + n] : v[i], give = up ? v[i] : v[i + n];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// The tables of the C = T*K <= 256 routed pairs (expert ids in ids_s), by one CTA: stable sort by expert, list of the
// experts with work and their work records. A pair's column is the number of pairs in front of it, which its
// threads count directly (a scan over 256 experts was most of the time of this step).
__device__ __forceinline__ void decode_tables(const RouteDev& R, const int* ids_s, int C, int E, int K, unsigned* mask_s, int* c0_s) {
    const int tid = threadIdx.x;
    if (tid < MAX_EXPERTS / 32) mask_s[tid] = 0u;
    __syncthreads();
    // four threads per pair at up to 128 pairs, two above; each takes every 4th (2nd) quadruple of pairs
    const int sh = (C <= RS_THREADS / 4) ? 2 : 1, per = 1 << sh, part = tid & (per - 1), p = tid >> sh;
    const int e = (p < C) ? ids_s[p] : 0;
    if (p < C && part == 0) atomicOr(&mask_s[e >> 5], 1u << (e & 31));
    int less = 0, before = 0, same = 0;  // smaller experts; same expert, lower pair; same expert
    if (p < C) {
#pragma unroll 2
        for (int q = part * 4; q < C; q += per * 4) {
            const int4 v = *reinterpret_cast<const int4*>(&ids_s[q]);  // (padded with ids no expert has)
            const int x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                less += x[i] < e;
                same += x[i] == e;
                before += (x[i] == e) && (q + i < p);
            }
        }
    }
    for (int o = 1; o < per; o <<= 1) {
        less += __shfl_xor_sync(0xffffffffu, less, o);
        same += __shfl_xor_sync(0xffffffffu, same, o);
        before += __shfl_xor_sync(0xffffffffu, before, o);
    }
    __syncthreads();
    auto rank_of = [&](int ex) {  // experts with work below ex
        int u = 0;
#pragma unroll
        for (int w = 0; w < MAX_EXPERTS / 32; ++w) {
            const unsigned m = mask_s[w];
            u += (w < (ex >> 5)) ? __popc(m) : (w == (ex >> 5)) ? __popc(m & ((1u << (ex & 31)) - 1u)) : 0;
        }
        return u;
    };
    const int U = rank_of(MAX_EXPERTS - 1) + (int)(mask_s[MAX_EXPERTS / 32 - 1] >> 31);
    if (p < C && part == 0) {
        const int col = less + before, u = rank_of(e), tok = p / K;
        R.col_expert[col] = e;
        R.col_src_tok[col] = tok;
        R.dst_to_col[p] = col;
        // source tokens of the expert's first four columns ride in its work record, which a consumer
        // CTA reads in a single round trip {expert, first column, columns}
        if (before < 4) reinterpret_cast<int*>(R.work)[8 * u + 4 + before] = tok;
        if (before == 0) {
            R.work[2 * u] = make_int4(e, less, same, 0);
            R.uexp[u] = e;
            c0_s[u] = less;
        }
    }
    if (tid == 0) *R.n_uexp = U;
    const int nu_max = (C < E) ? C : E;
    if (tid >= U && tid < nu_max) R.work[2 * tid] = make_int4(-1, 0, 0, 0);
    __syncthreads();
    if (tid <= E) {
        // bound of expert tid: first column of the next expert with work
        const int u = (tid < MAX_EXPERTS) ? rank_of(tid) : U;
        R.expert_bounds[tid] = (u < U) ? c0_s[u] : C;
    }
}

// Router of a decode batch. The first CTAs: the logits of an expert row (or two) for all tokens; the CTAs after them: the
// activation operand (and the normed activations), one token and RS_BLOCKS blocks each; the last
// CTA to finish (fence + ticket, no spin) routes: one warp per token, then the tables.
// Bound by the chain of dependent steps, so each of them is as short as it goes: all tokens' inputs of a thread are
// requested together, the fused RMSNorm needs no pass of its own (a logit is scaled by its token's
// 1 / rms after the sum, whose squares ride along), sixteen sums cross the warp in 16 shuffles. (One token after
// the other, with a shared two-term reduction each, this kernel took 25 us at 16 tokens; now ~10.)
// ROWS: expert rows of a logit CTA: two for 256 experts, so that the CTAs (one per SM: 128 registers a thread) are one wave.
template <int NS, int ROWS>  // NS * 32 >= E
__global__ void __launch_bounds__(RS_THREADS)
router_small_kernel(const __grid_constant__ DecodeArgs a, const int logit_ctas, const int parts) {
    __shared__ float red_s[ROWS][RS_WARPS][DECODE_MAX_TOKENS], ssq_s[RS_WARPS][DECODE_MAX_TOKENS];
    __shared__ __align__(16) float p_s[RS_WARPS][NS * 32];
    __shared__ __align__(16) int ids_s[DECODE_MAX_TOKENS * MAX_TOP_K];
    __shared__ int c0_s[MAX_EXPERTS];
    __shared__ unsigned mask_s[MAX_EXPERTS / 32];
    __shared__ int is_last_s;
    __shared__ unsigned long long tab_s[32];

    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int H = a.L.H, E = a.L.E, T = a.T, K = a.K;
    const int H4 = H >> 2;
    const bool is_logit = (int)blockIdx.x < logit_ctas;
    if (tid < 32) tab_s[tid] = lumen_exact::exp2_tab_entry(tid);

    if (is_logit) {
        const int e0 = blockIdx.x * ROWS;
        const float4* wrow[ROWS];
        float4 w4[ROWS];
        // first part of the router rows in registers before waiting on the previous kernel (weights are static)
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            wrow[r] = reinterpret_cast<const float4*>(a.L.router_w + (size_t)min(e0 + r, E - 1) * H);
            w4[r] = (tid < H4) ? __ldg(wrow[r] + tid) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        pdl_wait();
        float acc[ROWS][DECODE_MAX_TOKENS], sq[DECODE_MAX_TOKENS];
#pragma unroll
        for (int t = 0; t < DECODE_MAX_TOKENS; ++t) {
            sq[t] = 0.0f;
#pragma unroll
            for (int r = 0; r < ROWS; ++r) acc[r][t] = 0.0f;
        }
#pragma unroll 1
        for (int i4 = tid; i4 < H4; i4 += RS_THREADS) {
            if (i4 != tid) {
#pragma unroll
                for (int r = 0; r < ROWS; ++r) w4[r] = __ldg(wrow[r] + i4);
            }
            if (a.gamma != nullptr) {
                const float4 g = __ldg(reinterpret_cast<const float4*>(a.gamma) + i4);
#pragma unroll
                for (int r = 0; r < ROWS; ++r) w4[r] = make_float4(w4[r].x * g.x, w4[r].y * g.y, w4[r].z * g.z, w4[r].w * g.w);
            }
            constexpr int TB = DECODE_MAX_TOKENS / ROWS;  // tokens whose inputs are in flight together
#pragma unroll
            for (int t0 = 0; t0 < DECODE_MAX_TOKENS; t0 += TB) {
                float4 xv[TB];
#pragma unroll
                for (int t = 0; t < TB; ++t)
                    if (t0 + t < T) xv[t] = reinterpret_cast<const float4*>(a.x + (size_t)(t0 + t) * H)[i4];
#pragma unroll
                for (int t = 0; t < TB; ++t)
                    if (t0 + t < T) {
#pragma unroll
                        for (int r = 0; r < ROWS; ++r)
                            acc[r][t0 + t] += w4[r].x * xv[t].x + w4[r].y * xv[t].y + w4[r].z * xv[t].z + w4[r].w * xv[t].w;
                        if (a.gamma != nullptr)
                            sq[t0 + t] += xv[t].x * xv[t].x + xv[t].y * xv[t].y + xv[t].z * xv[t].z + xv[t].w * xv[t].w;
                    }
            }
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const float v = warp_sum16(acc[r]);
            if ((lane & 1) == 0) red_s[r][warp][lane >> 1] = v;
        }
        if (a.gamma != nullptr) {
            const float q = warp_sum16(sq);
            if ((lane & 1) == 0) ssq_s[warp][lane >> 1] = q;
        }
        __syncthreads();
        const int tt = tid & (DECODE_MAX_TOKENS - 1), rr = tid / DECODE_MAX_TOKENS;
        if (rr < ROWS && tt < T && e0 + rr < E) {
            float sum = 0.0f, ss = 0.0f;
#pragma unroll
            for (int w = 0; w < RS_WARPS; ++w) sum += red_s[rr][w][tt];
            if (a.gamma != nullptr) {
#pragma unroll
                for (int w = 0; w < RS_WARPS; ++w) ss += ssq_s[w][tt];
                sum *= 1.0f / sqrtf(ss / (float)H + a.eps);
            }
            a.R.logits[(size_t)tt * E + e0 + rr] = sum;
        }
    } else if (parts > 0) {
        // activation operand of the gate/up kernel (and the normed output of the fused-norm entry
        // point): two-term int8 blocks for Q4_0 weights, 16-bit hi + lo fragments otherwise
        const int o = blockIdx.x - logit_ctas, t = o / parts, b = (o - t * parts) * RS_BLOCKS + (tid >> 3);
        const int nblk = H >> 5, nblk_pad = a.L.kg_h * 4, sub = tid & 7;
        const float4* xr = reinterpret_cast<const float4*>(a.x + (size_t)t * H);
        pdl_wait();
        float scale = 1.0f;
        if (a.gamma != nullptr) {
            float ss = 0.0f;
            for (int i4 = tid; i4 < H4; i4 += RS_THREADS) {
                const float4 v = xr[i4];
                ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
            }
#pragma unroll
            for (int k = 16; k > 0; k >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, k);
            if (lane == 0) ssq_s[warp][0] = ss;
            __syncthreads();
            ss = 0.0f;
#pragma unroll
            for (int w = 0; w < RS_WARPS; ++w) ss += ssq_s[w][0];
            scale = 1.0f / sqrtf(ss / (float)H + a.eps);
        }
        auto load_x4 = [&](int i4) -> float4 {
            float4 v = xr[i4];
            if (a.gamma != nullptr) {
                const float4 g = __ldg(reinterpret_cast<const float4*>(a.gamma) + i4);
                v.x = v.x * scale * g.x;
                v.y = v.y * scale * g.y;
                v.z = v.z * scale * g.z;
                v.w = v.w * scale * g.w;
            }
            return v;
        };
        if (b < nblk) {  // (the eight lanes of a block agree)
            float4* normed = (a.gamma != nullptr && a.normed_out != nullptr) ? reinterpret_cast<float4*>(a.normed_out + (size_t)t * H) : nullptr;
            if (a.xq != nullptr) {
                const float4 v = load_x4(b * 8 + sub);
                dcommon::build_xq_block(v, sub, lane, a.xq + (size_t)t * dcommon::xq_tok_words(nblk_pad), nblk_pad, b);
                if (normed) normed[b * 8 + sub] = v;
            } else {
                const int hl = sub >> 2, t4 = sub & 3;
                const float4 lo4 = load_x4(b * 8 + t4), hi4 = load_x4(b * 8 + 4 + t4);
                a.xf[((size_t)(t * 2 + hl) * nblk_pad + b) * 4 + t4] = make_act_frag(lo4, hi4, hl, a.L.quant == BF16);
                if (normed) normed[b * 8 + (hl ? 4 : 0) + t4] = hl ? hi4 : lo4;
            }
        }
    } else {
        pdl_wait();  // (logits supplied, no operand wanted: this CTA only routes)
    }

    // last-CTA election: the CTA barrier orders every thread's stores before
    // thread 0's device-scope fence and ticket (fences are cumulative)
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        const unsigned int ticket = atomicAdd(a.R.ticket, 1u);
        is_last_s = (ticket == gridDim.x - 1);
        if (is_last_s) __threadfence();
    }
    __syncthreads();
    if (!is_last_s) return;

    const float* lg = (a.logits_override == nullptr) ? a.R.logits : a.logits_override;
    if (tid < DECODE_MAX_TOKENS * MAX_TOP_K) ids_s[tid] = 0x7fffffff;  // padding: an id no expert has
    __syncthreads();
    if (warp < T) {
        float v[NS];
#pragma unroll
        for (int i = 0; i < NS; ++i) v[i] = (lane + 32 * i < E) ? __ldcg(lg + (size_t)warp * E + lane + 32 * i) : -INFINITY;
        int id;
        const float w = warp_route<NS>(v, E, K, a.gating, p_s[warp], reinterpret_cast<const uint64_t*>(tab_s), id);
        if (lane < K) {
            a.R.ids[(size_t)warp * K + lane] = (uint32_t)id;
            a.R.weights[(size_t)warp * K + lane] = w;
            ids_s[warp * K + lane] = id;
        }
    }
    __syncthreads();
    decode_tables(a.R, ids_s, T * K, E, K, mask_s, c0_s);
    if (tid == 0) *a.R.ticket = 0u;
}

// ---------------------------------------------------------------------------
// gate/up + SwiGLU
// ---------------------------------------------------------------------------
constexpr int GU_THREADS = 256;
constexpr int GU_WARPS = GU_THREADS / 32;

// NG: column groups the code covers (1 or 4). The groups' bodies are predicated, not branched
// around, so a caller that knows there is one group uses NG = 1 and issues a quarter of the code.
template <int Q, int NG = 4>
__device__ __forceinline__ void tile_mma_pair(const WTile<Q>& wg, const WTile<Q>& wu,
                                              const uint4* (&bptr)[4], int ngroups,
                                              float (&acc_g)[4][4], float (&acc_u)[4][4]) {
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        uint32_t g_lo[4], g_hi[4], u_lo[4], u_hi[4];
        unpack_block<Q>(wg, b, g_lo, g_hi);
        unpack_block<Q>(wu, b, u_lo, u_hi);
        const float2 sg = block_scales<Q>(wg, b);
        const float2 su = block_scales<Q>(wu, b);
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            if (g < ngroups) {
                uint4 bf = make_uint4(0u, 0u, 0u, 0u);
                if (bptr[g] != nullptr) bf = ldg_cached(bptr[g] + b * 4);
                float cg[4] = {0.f, 0.f, 0.f, 0.f}, cu[4] = {0.f, 0.f, 0.f, 0.f};
                if (Q == BF16) {
                    mma_bf16(cg, g_lo, bf.x, bf.y);
                    mma_bf16(cg, g_hi, bf.z, bf.w);
                    mma_bf16(cu, u_lo, bf.x, bf.y);
                    mma_bf16(cu, u_hi, bf.z, bf.w);
                } else {
                    mma_f16(cg, g_lo, bf.x, bf.y);
                    mma_f16(cg, g_hi, bf.z, bf.w);
                    mma_f16(cu, u_lo, bf.x, bf.y);
                    mma_f16(cu, u_hi, bf.z, bf.w);
                }
                acc_g[g][0] = fmaf(sg.x, cg[0], acc_g[g][0]);
                acc_g[g][1] = fmaf(sg.x, cg[1], acc_g[g][1]);
                acc_g[g][2] = fmaf(sg.y, cg[2], acc_g[g][2]);
                acc_g[g][3] = fmaf(sg.y, cg[3], acc_g[g][3]);
                acc_u[g][0] = fmaf(su.x, cu[0], acc_u[g][0]);
                acc_u[g][1] = fmaf(su.x, cu[1], acc_u[g][1]);
                acc_u[g][2] = fmaf(su.y, cu[2], acc_u[g][2]);
                acc_u[g][3] = fmaf(su.y, cu[3], acc_u[g][3]);
            }
        }
    }
}

template <int Q>
__global__ void __launch_bounds__(GU_THREADS)
gate_up_kernel(const __grid_constant__ DecodeArgs a) {
    __shared__ float red[GU_WARPS][4][16][4][2];  // [warp][group][row][token in group][gate,up]
    // wait first, then release the down kernel: it reads the router's tables before its own wait
    pdl_wait();
    pdl_trigger();
    const int u = blockIdx.y;
    if (u >= *a.R.n_uexp) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gq = lane >> 2, t4 = lane & 3;
    const int rt = blockIdx.x;
    const int e = a.R.uexp[u];
    const int c0 = a.R.expert_bounds[e], c1 = a.R.expert_bounds[e + 1];
    const int kg_h = a.L.kg_h, I = a.L.I;
    const int nblk_pad = kg_h * 4, nblk_i_pad = a.L.kg_i * 4;
    const uint4* gq_base = a.L.gate_q(e);
    const uint4* uq_base = a.L.up_q(e);
    const uint4* gs_base = a.L.gate_s(e);
    const uint4* us_base = a.L.up_s(e);

    for (int chunk = c0; chunk < c1; chunk += 16) {
        const int ncol = min(16, c1 - chunk);
        const int ng = (ncol + 3) >> 2;
        const uint4* bbase[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const int col = chunk + 4 * g + (gq >> 1);
            bbase[g] = nullptr;
            if (g < ng && col < c1) {
                const int tok = a.R.col_src_tok[col];
                bbase[g] = a.xf + ((size_t)(tok * 2 + (gq & 1)) * nblk_pad) * 4 + t4;
            }
        }
        float acc_g[4][4], acc_u[4][4];
#pragma unroll
        for (int g = 0; g < 4; ++g)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc_g[g][i] = acc_u[g][i] = 0.0f;

        WTile<Q> wg, wu, ng_t, nu_t;
        int kg = warp;
        if (kg < kg_h) {
            load_wtile<Q>(wg, gq_base, gs_base, rt * kg_h + kg, lane);
            load_wtile<Q>(wu, uq_base, us_base, rt * kg_h + kg, lane);
        }
        for (; kg < kg_h; kg += GU_WARPS) {
            const bool more = (kg + GU_WARPS) < kg_h;
            if (more) {
                load_wtile<Q>(ng_t, gq_base, gs_base, rt * kg_h + kg + GU_WARPS, lane);
                load_wtile<Q>(nu_t, uq_base, us_base, rt * kg_h + kg + GU_WARPS, lane);
            }
            const uint4* bp[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) bp[g] = bbase[g] ? bbase[g] + (size_t)kg * 16 : nullptr;
            if (ng <= 1) tile_mma_pair<Q, 1>(wg, wu, bp, ng, acc_g, acc_u);
            else tile_mma_pair<Q, 4>(wg, wu, bp, ng, acc_g, acc_u);
            if (more) {
                wg = ng_t;
                wu = nu_t;
            }
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            red[warp][g][gq][t4][0] = acc_g[g][0] + acc_g[g][1];
            red[warp][g][gq][t4][1] = acc_u[g][0] + acc_u[g][1];
            red[warp][g][gq + 8][t4][0] = acc_g[g][2] + acc_g[g][3];
            red[warp][g][gq + 8][t4][1] = acc_u[g][2] + acc_u[g][3];
        }
        __syncthreads();
        {
            const int row = tid & 15, tokc = tid >> 4;
            if (tokc < ncol) {
                float gate = 0.0f, up = 0.0f;
#pragma unroll
                for (int w = 0; w < GU_WARPS; ++w) {
                    gate += red[w][tokc >> 2][row][tokc & 3][0];
                    up += red[w][tokc >> 2][row][tokc & 3][1];
                }
                const float sv = (gate / (1.0f + expf(-gate))) * up;
                const int col = chunk + tokc;
                const int irow = rt * 16 + row;
                if (a.s_f32 != nullptr) a.s_f32[(size_t)col * I + irow] = sv;
                dcommon::store_swiglu_frag<Q>(a.sf, col, irow, nblk_i_pad, sv);
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// down projection for any number of columns per expert (mma.sync grouped path of
// the prefill entry point): one CTA per (16 rows of H, expert), k-groups split
// across warps, output f16 by compact column for the scatter-accumulate.
// ---------------------------------------------------------------------------
template <int Q>
__global__ void __launch_bounds__(GU_THREADS)
down_general_kernel(const __grid_constant__ DecodeArgs a, __half* __restrict__ d16) {
    __shared__ float red[GU_WARPS][4][16][4];
    const int u = blockIdx.y;
    if (u >= *a.R.n_uexp) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gq = lane >> 2, t4 = lane & 3;
    const int rt = blockIdx.x;
    const int e = a.R.uexp[u];
    const int c0 = a.R.expert_bounds[e], c1 = a.R.expert_bounds[e + 1];
    const int kg_i = a.L.kg_i, H = a.L.H;
    const int nblk_i_pad = kg_i * 4;
    const uint4* q_base = a.L.down_q(e);
    const uint4* s_base = a.L.down_s(e);
    for (int chunk = c0; chunk < c1; chunk += 16) {
        const int ncol = min(16, c1 - chunk);
        const int ng = (ncol + 3) >> 2;
        const uint4* bbase[4];
        float acc[4][4];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const int colr = 4 * g + (gq >> 1);
            bbase[g] = (colr < ncol)
                           ? a.sf + ((size_t)((chunk + colr) * 2 + (gq & 1)) * nblk_i_pad) * 4 + t4
                           : nullptr;
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[g][i] = 0.0f;
        }
        for (int kg = warp; kg < kg_i; kg += GU_WARPS) {
            WTile<Q> w;
            load_wtile<Q>(w, q_base, s_base, rt * kg_i + kg, lane);
            const uint4* bp[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) bp[g] = bbase[g] ? bbase[g] + (size_t)kg * 16 : nullptr;
            tile_mma<Q, 4>(w, bp, ng, acc);
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            red[warp][g][gq][t4] = acc[g][0] + acc[g][1];
            red[warp][g][gq + 8][t4] = acc[g][2] + acc[g][3];
        }
        __syncthreads();
        {
            const int row = tid & 15, tokc = tid >> 4;
            if (tokc < ncol) {
                float v = 0.0f;
#pragma unroll
                for (int w = 0; w < GU_WARPS; ++w) v += red[w][tokc >> 2][row][tokc & 3];
                d16[(size_t)(chunk + tokc) * H + rt * 16 + row] = __float2half_rn(v);
            }
        }
        __syncthreads();
    }
}

cudaError_t launch_grouped_mma(const DecodeArgs& a, __half* d16, cudaStream_t st) {
    const dim3 g_gu(a.L.rt_i, a.L.E), g_dn(a.L.rt_h, a.L.E);
    count_launch(2);
    switch (a.L.quant) {
        case Q4_0:
            gate_up_kernel<Q4_0><<<g_gu, GU_THREADS, 0, st>>>(a);
            down_general_kernel<Q4_0><<<g_dn, GU_THREADS, 0, st>>>(a, d16);
            break;
        case Q8_0:
            gate_up_kernel<Q8_0><<<g_gu, GU_THREADS, 0, st>>>(a);
            down_general_kernel<Q8_0><<<g_dn, GU_THREADS, 0, st>>>(a, d16);
            break;
        default:
            gate_up_kernel<BF16><<<g_gu, GU_THREADS, 0, st>>>(a);
            down_general_kernel<BF16><<<g_dn, GU_THREADS, 0, st>>>(a, d16);
            break;
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// launch
// ---------------------------------------------------------------------------
cudaError_t launch_route_small(const DecodeArgs& a, cudaStream_t st) {
    const int rows = (a.L.E > 128) ? 2 : 1;
    const int logit_ctas = (a.logits_override == nullptr) ? (a.L.E + rows - 1) / rows : 0;
    const int parts = (a.xq != nullptr || a.xf != nullptr) ? (a.L.H / 32 + RS_BLOCKS - 1) / RS_BLOCKS : 0;
    const int grid = logit_ctas + a.T * parts;
    count_launch();
    auto go = [&](auto kern) {
        return launch_dep(kern, dim3(grid > 0 ? grid : 1), dim3(RS_THREADS), 0, st, a, logit_ctas, parts);
    };
    return (a.L.E <= 32) ? go(router_small_kernel<1, 1>) : (a.L.E <= 128) ? go(router_small_kernel<4, 1>) : go(router_small_kernel<8, 2>);
}

bool decode_stream_applicable(const DecodeArgs& a);
cudaError_t launch_gate_up_stream(const DecodeArgs& a, cudaStream_t st);

cudaError_t launch_decode_phase(const DecodeArgs& a_in, int phase, bool alone, cudaStream_t st) {
    DecodeArgs a = a_in;
    // Q4_0 layers that gate_up_stream_kernel takes: int8 activations for both products; every other format and shape:
    // hi + lo fragments and the general streaming kernel
    // (up to three tokens only where the context asks for the chain: the fused kernel, which such a batch takes
    // otherwise, gives the down product the finer activations)
    const bool int8 = decode_stream_applicable(a) && (a.T >= 4 || a.bar == nullptr);
    if (!int8) a.xq = a.sq = nullptr;
    if (phase == 0) return launch_route_small(a, st);
    if (phase == 1) return int8 ? launch_gate_up_stream(a, st) : launch_stream_gate_up(a, st);
    return launch_stream_down(a, int8, !alone, st);
}

bool decode_fused_applicable(const DecodeArgs& a);
cudaError_t launch_decode_fused(const DecodeArgs& a, cudaStream_t st);

// Which form a decode call takes: the persistent fused kernel (two grid barriers, no boundary between kernels) is ahead
// while the weights of the selected experts are so few that boundaries cost more than streaming them; the chain's
// kernels stream faster. Measured us per call, fused / chain, at H = 2048, I = 768, E = 128, top-8 (40 MB Q8_0, 75 MB
// BF16 per token): Q8_0 32.8 / 33.7 at two tokens, 41.2 / 39.7 at three; BF16 32.6 / 29.7 at one, 66 / 38 at two; at
// H = 1024, I = 512, top-6: Q8_0 24.0 / 23.6 at three, BF16 24.8 / 22.1 at two. Q4_0: fused up to three tokens (32.8 us
// at three; with activations as fine as its own the chain takes 33.7), the int8 chain from four (38 / 31 us). One expert:
// always fused where it applies (four tokens of Q4_0 13.2 us, the chain 19.4).
bool decode_uses_fused(const DecodeArgs& a) {
    if (!decode_fused_applicable(a)) return false;
    if (a.L.E == 1) return true;
    const double weights = 3.0 * a.T * a.K * a.L.I * a.L.H;
    switch (a.L.quant) {
        case Q4_0: return a.T < 4 || !decode_stream_applicable(a);
        case Q8_0: return a.T < 3 || weights * (34.0 / 32) < 28e6;
        default: return weights * 2 < (a.T < 2 ? 60e6 : 36e6);
    }
}

cudaError_t launch_decode(const DecodeArgs& a, cudaStream_t st) {
    if (decode_uses_fused(a)) return launch_decode_fused(a, st);
    for (int phase = 0; phase < 3; ++phase) {
        const cudaError_t err = launch_decode_phase(a, phase, false, st);
        if (err != cudaSuccess) return err;
    }
    return cudaSuccess;
}

}  // namespace lumen
