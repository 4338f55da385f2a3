// Routing and dispatch tables for multi-token batches (prefill), entirely on the
// device: the reference does this part of encode_moe_ffn_prefill_grouped with a
// blocking device-to-host copy, a host loop and four to six uploads per layer
// (crates/lumen-runtime/src/cuda/moe.rs:2105-2207).
//
//   router_logits_large_kernel  logits[T,E] = X[T,H] W_r[E,H]^T, f32 accumulate
//                               (moe_router_logits_batched, cuda/shaders/moe_grouped.cu:79)
//   topk_large_kernel           one warp per token (router.cuh)
//   route_single_kernel         contexts of one expert: everything up to the plan in one pass
//   sort_one_kernel (up to 2048 pairs), sort_hist / sort_rowscan / sort_place
//                               stable counting sort of (token, slot) pairs by
//                               expert, tokens ascending then slots ascending:
//                               expert_bounds, col_expert, col_src_tok, dst_to_col
//                               exactly as cuda/moe.rs:2115-2147; and
//                               the list of experts with work and the tile lists
//                               of the grouped GEMMs (cuda/moe.rs:2188-2207).
//   scatter_accum_kernel        out[t] = residual[t] + sum_slot w[t,slot] * D[dst_to_col[t,slot]]
//                               in slot order (moe_grouped_scatter_accum_q8_0,
//                               cuda/shaders/moe_grouped.cu:493-517).
#include "moe_internal.cuh"
#include "router.cuh"
#include "mma_frag.cuh"

#define CUDA_RET(expr)                         \
    do {                                       \
        const cudaError_t e_ = (expr);         \
        if (e_ != cudaSuccess) return e_;      \
    } while (0)

namespace lumen {

// ---------------------------------------------------------------------------
// logits: 64 tokens x 64 experts per CTA, BK = 32, 256 threads, 4x4 per thread
// ---------------------------------------------------------------------------
template <typename XT>
__device__ __forceinline__ float x_to_f32(XT v);
template <>
__device__ __forceinline__ float x_to_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float x_to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float x_to_f32<__half>(__half v) { return __half2float(v); }

template <typename XT>
__global__ void __launch_bounds__(256)
router_logits_large_kernel(const XT* __restrict__ x, const float* __restrict__ w, float* __restrict__ logits,
                           int T, int H, int E) {
    constexpr int BM = 64, BN = 64, BK = 32;
    __shared__ float xs[BK][BM + 1];
    __shared__ float ws[BK][BN + 1];
    const int tid = threadIdx.x;
    const int t0 = blockIdx.x * BM, e0 = blockIdx.y * BN;
    const int tx = tid & 15, ty = tid >> 4;  // tx: experts, ty: tokens
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    for (int k0 = 0; k0 < H; k0 += BK) {
        for (int i = tid; i < BM * BK; i += 256) {
            const int r = i / BK, c = i % BK;
            const int t = t0 + r;
            xs[c][r] = (t < T) ? x_to_f32<XT>(x[(size_t)t * H + k0 + c]) : 0.0f;
        }
        for (int i = tid; i < BN * BK; i += 256) {
            const int r = i / BK, c = i % BK;
            const int e = e0 + r;
            ws[c][r] = (e < E) ? w[(size_t)e * H + k0 + c] : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float xv[4], wv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) xv[i] = xs[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) wv[j] = ws[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xv[i], wv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = t0 + ty * 4 + i;
        if (t >= T) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int e = e0 + tx * 4 + j;
            if (e < E) logits[(size_t)t * E + e] = acc[i][j];
        }
    }
}

// ---------------------------------------------------------------------------
// logits on the tensor cores with f32-grade accuracy: X and W_r are each split into
// a high and a low f16 part and up to three m16n8k16 products (hi*hi + hi*lo + lo*hi)
// are accumulated in f32; the dropped lo*lo term is ~2^-22 relative. W_r is split
// once per call into two [E,H] f16 planes; X is split in registers (the lo*hi
// product is skipped for a fragment whose low parts are all zero, which is the
// usual case for bf16 activations).
// CTA = 64 tokens x (up to) 64 experts, 4 warps of 16 tokens (small tiles: at a few
// thousand tokens the grid must still cover the SMs). Per 32-input slab
// lane (g,t) owns inputs 8t..8t+7 of token rows g and g+8 (one 16-byte load each
// for bf16) and of expert row 8n+g (one 16-byte shared load per plane): the same
// input -> k-slot assignment on both operands, so the contraction is unchanged.
// ---------------------------------------------------------------------------
__global__ void split_router_w_kernel(const float* __restrict__ w, __half* __restrict__ w16, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v = w[i];
    const __half hi = __float2half_rn(v);
    w16[i] = hi;
    w16[n + i] = __float2half_rn(v - __half2float(hi));
}

__device__ __forceinline__ void cp_async16_rl(void* smem_dst, const void* gsrc) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gsrc) : "memory");
}

template <typename XT>
struct XSlab;  // 8 consecutive inputs of one token row
template <>
struct XSlab<__nv_bfloat16> {
    uint4 v;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { v = *reinterpret_cast<const uint4*>(p); }
    __device__ __forceinline__ void get(float* f) const {
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[2 * i] = __uint_as_float(u[i] << 16);
            f[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
        }
    }
};
template <>
struct XSlab<float> {
    float4 a, b;
    __device__ __forceinline__ void load(const float* p) {
        a = *reinterpret_cast<const float4*>(p);
        b = *reinterpret_cast<const float4*>(p + 4);
    }
    __device__ __forceinline__ void get(float* f) const {
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
        f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    }
};

__device__ __forceinline__ void split_pair(float v0, float v1, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(v0, v1);
    const float2 hf = __half22float2(h);
    const __half2 l = __floats2half2_rn(v0 - hf.x, v1 - hf.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// NE = experts per CTA: 64, or 32 for batches that would otherwise leave most SMs with a few warps
template <typename XT, int NE>
__global__ void __launch_bounds__(128)
router_logits_mma_kernel(const XT* __restrict__ x, const __half* __restrict__ w16, float* __restrict__ logits,
                         int T, int H, int E) {
    constexpr int BM = 64, BK = 32;
    // [buffer][plane][expert row][32 inputs]: 64-byte rows, 16-byte fragment loads are conflict-free
    __shared__ __align__(16) __half ws[2][2][NE][BK];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const int t0 = blockIdx.x * BM, e0 = blockIdx.y * NE;
    const int ne = min(NE, E - e0);
    const int ntile = (ne + 7) >> 3;
    const size_t plane = (size_t)E * H;
    float acc[NE / 8][4];
#pragma unroll
    for (int n = 0; n < NE / 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] = 0.0f;
    const int ra = t0 + warp * 16 + g, rb = ra + 8;
    const XT* xa = x + (size_t)min(ra, T - 1) * H + 8 * t4;
    const XT* xb = x + (size_t)min(rb, T - 1) * H + 8 * t4;
    auto stage_w = [&](int buf, int k0) {
        // NE rows x 4 chunks x 2 planes = 512 16-byte copies, 4 per thread
#pragma unroll
        for (int i = 0; i < NE / 16; ++i) {
            const int c = tid + i * 128;
            const int pl = c / (NE * 4), row = (c >> 2) % NE, ch = c & 3;
            const __half* src = w16 + pl * plane + (size_t)min(e0 + row, E - 1) * H + k0 + ch * 8;
            cp_async16_rl(&ws[buf][pl][row][ch * 8], src);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int nslab = H / BK;
    XSlab<XT> na, nb;
    stage_w(0, 0);
    na.load(xa);
    nb.load(xb);
    for (int sidx = 0; sidx < nslab; ++sidx) {
        const int buf = sidx & 1;
        XSlab<XT> ca = na, cb = nb;
        if (sidx + 1 < nslab) {
            stage_w(buf ^ 1, (sidx + 1) * BK);
            na.load(xa + (sidx + 1) * BK);
            nb.load(xb + (sidx + 1) * BK);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        float fa[8], fb[8];
        ca.get(fa);
        cb.get(fb);
        uint32_t ah[2][4], al[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            split_pair(fa[4 * j], fa[4 * j + 1], ah[j][0], al[j][0]);
            split_pair(fb[4 * j], fb[4 * j + 1], ah[j][1], al[j][1]);
            split_pair(fa[4 * j + 2], fa[4 * j + 3], ah[j][2], al[j][2]);
            split_pair(fb[4 * j + 2], fb[4 * j + 3], ah[j][3], al[j][3]);
        }
        uint32_t lo_or = 0;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) lo_or |= al[j][i];
        const bool use_lo = __any_sync(0xffffffffu, (lo_or & 0x7fff7fffu) != 0);
#pragma unroll
        for (int n = 0; n < NE / 8; ++n) {
            if (n < ntile) {
                const uint4 bh = *reinterpret_cast<const uint4*>(&ws[buf][0][n * 8 + g][8 * t4]);
                const uint4 bl = *reinterpret_cast<const uint4*>(&ws[buf][1][n * 8 + g][8 * t4]);
                if (use_lo) {
                    mma_f16(acc[n], al[0], bh.x, bh.y);
                    mma_f16(acc[n], al[1], bh.z, bh.w);
                }
                mma_f16(acc[n], ah[0], bl.x, bl.y);
                mma_f16(acc[n], ah[1], bl.z, bl.w);
                mma_f16(acc[n], ah[0], bh.x, bh.y);
                mma_f16(acc[n], ah[1], bh.z, bh.w);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int n = 0; n < NE / 8; ++n) {
        if (n < ntile) {
            const int ec = e0 + n * 8 + 2 * t4;
            if (ra < T) {
                if (ec < E) logits[(size_t)ra * E + ec] = acc[n][0];
                if (ec + 1 < E) logits[(size_t)ra * E + ec + 1] = acc[n][1];
            }
            if (rb < T) {
                if (ec < E) logits[(size_t)rb * E + ec] = acc[n][2];
                if (ec + 1 < E) logits[(size_t)rb * E + ec + 1] = acc[n][3];
            }
        }
    }
}

// Gating + top-k of a batch, one warp per token. NP > 0: the logits arrive as NP partial sums
// [NP][T][E] (k ranges of the tcgen05 router); they are added in a fixed order and the sum is left in
// logits_out. NP = 0: plain logits. NS * 32 >= E.
// A warp's chain of dependent steps is what this kernel costs (4096 tokens are 28 warps per SM), so
// all NS * NP logits of a lane are requested at once (one after the other they were 16 L2 round trips, two
// thirds of 22 us), and the exps of a lane are inline and independent of one another, their table
// in shared memory.
// blk_hist (null = none): the per-expert pair counts of this block's TK_WARPS tokens, the first
// step of the counting sort (one histogram per chunk of SORT_TOK = TK_WARPS tokens), written here
// instead of by a launch of its own.
constexpr int TK_WARPS = 8;
template <int NS, int NP>
__global__ void __launch_bounds__(TK_WARPS * 32)
topk_large_kernel(const float* __restrict__ logits, float* __restrict__ logits_out, int T, int E, int K,
                  int gating, uint32_t* __restrict__ ids, float* __restrict__ weights, int32_t* __restrict__ blk_hist) {
    __shared__ __align__(16) float p_s[TK_WARPS][NS * 32];
    __shared__ unsigned long long tab_s[32];
    __shared__ int h[NS * 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * TK_WARPS + warp;
    if (threadIdx.x < 32) tab_s[threadIdx.x] = lumen_exact::exp2_tab_entry(threadIdx.x);
    if (threadIdx.x < NS * 32) h[threadIdx.x] = 0;
    grid_dep_sync();
    __syncthreads();
    if (t < T) {
        constexpr int NL = NP > 0 ? NP : 1;
        float v[NL][NS];
#pragma unroll
        for (int q = 0; q < NL; ++q)
#pragma unroll
            for (int i = 0; i < NS; ++i) {
                const int e = lane + 32 * i;
                v[q][i] = (e < E) ? __ldg(&logits[((size_t)q * T + t) * E + e]) : -INFINITY;
            }
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            const int e = lane + 32 * i;
#pragma unroll
            for (int q = 1; q < NL; ++q) v[0][i] += v[q][i];
            if (NP > 0 && e < E) logits_out[(size_t)t * E + e] = v[0][i];
        }
        int id;
        const float w = warp_route<NS>(v[0], E, K, gating, p_s[warp], reinterpret_cast<const uint64_t*>(tab_s), id);
        if (lane < K) {
            ids[(size_t)t * K + lane] = (uint32_t)id;
            weights[(size_t)t * K + lane] = w;
            if (blk_hist != nullptr) atomicAdd(&h[id], 1);
        }
    }
    if (blk_hist == nullptr) return;
    __syncthreads();
    // layout [expert][chunk]: a warp of sort_rowscan then scans one expert's row with coalesced loads
    for (int e = threadIdx.x; e < E; e += TK_WARPS * 32) blk_hist[(size_t)e * gridDim.x + blockIdx.x] = h[e];
}

// ---------------------------------------------------------------------------
// stable counting sort
// ---------------------------------------------------------------------------
constexpr int SORT_TOK = TK_WARPS;  // tokens per chunk: one block of the top-k kernel; small chunks also spread the
                                   // placement (one warp per chunk) over the machine

__global__ void __launch_bounds__(256)
sort_hist_kernel(const uint32_t* __restrict__ ids, int T, int K, int E, int32_t* __restrict__ blk_hist) {
    grid_dep_sync();
    __shared__ int h[MAX_EXPERTS];
    const int tid = threadIdx.x;
    for (int e = tid; e < E; e += 256) h[e] = 0;
    __syncthreads();
    const int t0 = blockIdx.x * SORT_TOK;
    const int n = min(SORT_TOK, T - t0) * K;
    for (int p = tid; p < n; p += 256) atomicAdd(&h[ids[(size_t)t0 * K + p]], 1);
    __syncthreads();
    // layout [expert][chunk]: a warp of sort_rowscan then scans one expert's row with coalesced loads
    for (int e = tid; e < E; e += 256) blk_hist[(size_t)e * gridDim.x + blockIdx.x] = h[e];
}

// One warp per expert: exclusive scan over the chunk counts of the expert's row (in place);
// the row total goes behind the rows.
__global__ void __launch_bounds__(32)
sort_rowscan_kernel(int32_t* __restrict__ blk_hist, int nchunks) {
    grid_dep_sync();
    const int e = blockIdx.x, lane = threadIdx.x;
    int32_t* rowp = blk_hist + (size_t)e * nchunks;
    int run = 0;
    for (int c0 = 0; c0 < nchunks; c0 += 128) {
        int v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int c = c0 + u * 32 + lane;
            v[u] = (c < nchunks) ? rowp[c] : 0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int c = c0 + u * 32 + lane;
            int inc = v[u];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int w = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += w;
            }
            if (c < nchunks) rowp[c] = run + inc - v[u];
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
    }
    if (lane == 0) blk_hist[(size_t)gridDim.x * nchunks + e] = run;
}

// What the plan of a call consists of besides the sorted pairs: expert segment bounds and the tile
// lists of the expert products. tile entry: {expert, col_start, ncols, m_tile}.
struct PlanArgs {
    int E, tile_shift, tile_shift_dn, mt_gu, mt_dn;  // log2 of the columns per tile
    int4 *tiles_gu, *tiles_dn;
    int32_t* n_tiles;
    int max_tiles_gu, max_tiles_dn;
    int32_t* any_lo;    // the router's "some low part is non-zero" word: zeroed for the next call
    int32_t* starts;    // item shares of the streaming kernels (null = none)
    int ctas, rt_gu, rt_dn;
    // expert parallel: whether this call's work goes to the streaming kernels is known on the device only (null =
    // the lists above are what the host decided on); then their chunk list, and no tiles
    const int32_t* stream_mode;
    int4* chunks;
};

// By one CTA of PLAN_THREADS threads: plan from the experts' column counts in shared memory (E <= 256
// entries); bounds_s[0..E) receives the segment bounds.
// This runs once per call, alone, and every dependent instruction of its longest chain costs a few ns: the four
// scans run side by side on eight warps each (thread = expert), and so do the lists that follow. (One
// warp doing all scans with eight experts per lane took the one-CTA sort 9-12 us.)
constexpr int PLAN_THREADS = 1024;
__device__ __forceinline__ void emit_plan(const PlanArgs& a, const RouteDev& R, const int* cnt_s, int* bounds_s) {
    enum { COLS, TILES, TILES_DN, COST };  // TILES: chunks of the first list in the low, experts with work in the high half
    __shared__ int off_s[4][MAX_EXPERTS];  // exclusive sums over the experts
    __shared__ int tot_s[4];
    __shared__ __align__(16) int wsum_s[4][8];
    const int tid = threadIdx.x, lane = tid & 31, E = a.E;
    const int v = tid >> 8, e = tid & 255, wv = e >> 5;
    // the router's "some low part is non-zero" word, read by now, is zero again for the next call
    if (a.any_lo != nullptr && tid == 0) *a.any_lo = 0;
    if (tid >= 1022) a.n_tiles[2 + (tid & 1)] = 0;  // tile counters of the grouped products (tiles are claimed dynamically)
    const bool to_stream = a.stream_mode != nullptr && *a.stream_mode != 0;
    const bool to_tc = a.stream_mode != nullptr && !to_stream;
    const int tsh = to_stream ? STREAM_SHIFT : a.tile_shift, tc = 1 << tsh;
    // An item of the streaming kernels costs ~1 + n for a chunk of up to 8 n columns: unpacking the
    // weights, then every group of eight columns.
    const int full_cost = 1 + (tc >> 3);
    const int c = (e < E) ? cnt_s[e] : 0;
    int x = c;
    if (v == TILES) x = ((c + tc - 1) >> tsh) | (c > 0 ? 1 << 20 : 0);
    if (v == TILES_DN) x = (c + (1 << a.tile_shift_dn) - 1) >> a.tile_shift_dn;
    if (v == COST) {
        const int rest = c & (tc - 1);
        x = (c >> tsh) * full_cost + (rest ? 1 + ((rest + 7) >> 3) : 0);
    }
    int inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int w = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += w;
    }
    if (lane == 31) wsum_s[v][wv] = inc;
    __syncthreads();
    {
        const int4 s0 = *reinterpret_cast<const int4*>(&wsum_s[v][0]), s1 = *reinterpret_cast<const int4*>(&wsum_s[v][4]);
        const int ws[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
        int base = 0, total = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            base += (w < wv) ? ws[w] : 0;
            total += ws[w];
        }
        const int o = inc - x + base;
        off_s[v][e] = (v == TILES) ? o & 0xfffff : o;
        if (v == COLS && e < E) {
            R.expert_bounds[e] = o;
            bounds_s[e] = o;
        }
        if (v == TILES && c > 0) R.uexp[o >> 20] = e;
        if (e == 0) {
            tot_s[v] = (v == TILES) ? total & 0xfffff : total;
            if (v == COLS) R.expert_bounds[E] = total;
            if (v == TILES) *R.n_uexp = total >> 20;
            if (v == TILES) a.n_tiles[0] = to_stream ? 0 : min((total & 0xfffff) * a.mt_gu, a.max_tiles_gu);
            if (v == TILES_DN) a.n_tiles[1] = to_stream ? 0 : min(total * a.mt_dn, a.max_tiles_dn);
        }
    }
    __syncthreads();
    // largest expert with off[e] <= y (y below the total)
    auto expert_of = [&](const int* off, int y) {
        int lo = 0, hi = E;
#pragma unroll 1
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (off[mid] <= y) lo = mid;
            else hi = mid;
        }
        return lo;
    };
    if (v < 3) {
        // Column tiles in expert order: a thread takes column chunk q, finds its expert by bisection of the
        // chunk offsets, writes the chunk's m-tiles. The m-tile is the fastest index so that CTAs
        // running side by side share the same activation tile.
        const bool dn = (v == 2);
        int4* tiles = dn ? (to_stream ? nullptr : a.tiles_dn) : to_stream ? a.chunks : a.tiles_gu;
        const int* off = off_s[dn ? TILES_DN : TILES];
        const int total = tiles ? tot_s[dn ? TILES_DN : TILES] : 0;
        const int sh = dn ? a.tile_shift_dn : tsh, mt_n = dn ? a.mt_dn : to_stream ? 1 : a.mt_gu, max_tiles = dn ? a.max_tiles_dn : a.max_tiles_gu;
#pragma unroll 1
        for (int q = dn ? e : tid; q < total; q += dn ? 256 : 512) {
            const int ee = expert_of(off, q), ct = q - off[ee];
            const int cs = bounds_s[ee] + (ct << sh), nc = min(1 << sh, cnt_s[ee] - (ct << sh));
#pragma unroll 1
            for (int mt = 0, idx = q * mt_n; mt < mt_n && idx < max_tiles; ++mt, ++idx) tiles[idx] = make_int4(ee, cs, nc, mt);
        }
    } else if (a.starts != nullptr) {
        // shares of the streaming kernels' CTAs: contiguous item ranges of equal cost
        const float per_cta = (float)tot_s[COST] / (float)a.ctas;
#pragma unroll 1
        for (int i = e; i <= a.ctas; i += 256) {
            int chunk = to_tc ? 0 : tot_s[TILES];
            float frac = 0.0f;
            if (i < a.ctas && !to_tc) {
                const float want = per_cta * (float)i;
                const int ee = expert_of(off_s[COST], min((int)want, tot_s[COST] - 1));
                const float rest = want - (float)off_s[COST][ee];
                const int ct = (int)rest / full_cost;
                chunk = off_s[TILES][ee] + ct;
                frac = __fdividef(rest - (float)(ct * full_cost), (float)(1 + ((min(tc, cnt_s[ee] - (ct << tsh)) + 7) >> 3)));
            }
            a.starts[i] = chunk * a.rt_gu + min((int)(frac * (float)a.rt_gu), a.rt_gu);
            a.starts[a.ctas + 1 + i] = chunk * a.rt_dn + min((int)(frac * (float)a.rt_dn), a.rt_dn);
        }
    }
}

// One CTA: the plan of an expert-parallel call, from the totals left in expert_bounds.
__global__ void __launch_bounds__(PLAN_THREADS)
sort_scan_kernel(const __grid_constant__ PlanArgs a, RouteDev R) {
    grid_dep_sync();
    __shared__ int cnt_s[MAX_EXPERTS];
    __shared__ int bounds_s[MAX_EXPERTS];
    if (threadIdx.x < a.E) cnt_s[threadIdx.x] = R.expert_bounds[threadIdx.x];
    __syncthreads();
    emit_plan(a, R, cnt_s, bounds_s);
}

// The whole sort of a short batch (up to SORT1_MAX pairs) in one CTA: a warp owns a contiguous
// run of pairs, counts them per expert (lanes with the same expert find each other by a match, so no
// atomics), the counts are scanned over warps and experts, and the warp places its pairs. One
// launch for the three below: at 77 tokens they took 11 us of a 217 us call, this one 5.
constexpr int SORT1_MAX = 2048, SORT1_WARPS = PLAN_THREADS / 32;
__global__ void __launch_bounds__(SORT1_WARPS * 32)
sort_one_kernel(const uint32_t* __restrict__ ids, int C, int K, RouteDev R, const __grid_constant__ PlanArgs a) {
    __shared__ int wcnt[SORT1_WARPS * MAX_EXPERTS];  // [warp][E]
    __shared__ int cnt_s[MAX_EXPERTS];
    __shared__ int bounds_s[MAX_EXPERTS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, E = a.E;
    for (int i = tid; i < SORT1_WARPS * E; i += SORT1_WARPS * 32) wcnt[i] = 0;
    grid_dep_sync();
    __syncthreads();
    int* my = wcnt + warp * E;
    const int per = (C + SORT1_WARPS * 32 - 1) / (SORT1_WARPS * 32);  // 32-pair steps of a warp
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
#pragma unroll 1
        for (int i = 0; i < per; ++i) {
            const int p = (warp * per + i) * 32 + lane;
            const int e = (p < C) ? (int)ids[p] : -1 - lane;  // padding lanes match nobody
            const unsigned same = __match_any_sync(0xffffffffu, e), below = same & ((1u << lane) - 1u);
            if (pass == 1 && e >= 0) {
                const int col = bounds_s[e] + my[e] + __popc(below);
                R.col_expert[col] = e;
                R.col_src_tok[col] = p / K;
                R.dst_to_col[p] = col;
            }
            __syncwarp();
            if (e >= 0 && below == 0u) my[e] += __popc(same);  // one leader per expert
            __syncwarp();
        }
        if (pass == 1) break;
        __syncthreads();
        if (tid < E) {
            int run = 0;
#pragma unroll 4
            for (int w = 0; w < SORT1_WARPS; ++w) {
                const int c = wcnt[w * E + tid];
                wcnt[w * E + tid] = run;
                run += c;
            }
            cnt_s[tid] = run;
        }
        __syncthreads();
        emit_plan(a, R, cnt_s, bounds_s);
        __syncthreads();
    }
}

// A context of one expert (the always-on shared expert): there is nothing to rank or sort. One warp per token: the gate
// logit in f32, the weight, the identity tables and, in the same pass over the row, the f16 operand plane; the first CTA
// also writes the plan. It takes the place of the five kernels of the general chain: with the gather that goes too, the
// shared expert of 300 tokens takes 47 us instead of 64.
// x2f: 4 inputs as f32.
template <typename XT>
__device__ __forceinline__ float4 x2f(const XT* p);
template <>
__device__ __forceinline__ float4 x2f<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <>
__device__ __forceinline__ float4 x2f<__nv_bfloat16>(const __nv_bfloat16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                       __uint_as_float(u.y & 0xffff0000u));
}

template <typename XT>
__global__ void __launch_bounds__(256)
route_single_kernel(const XT* __restrict__ x, const float* __restrict__ w, int T, int H, int gating, RouteDev R,
                    __half* __restrict__ plane, bool natural, const __grid_constant__ PlanArgs plan) {
    __shared__ unsigned long long tab_s[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * 8 + warp;
    if (threadIdx.x < 32) tab_s[threadIdx.x] = lumen_exact::exp2_tab_entry(threadIdx.x);
    grid_dep_sync();
    __syncthreads();
    if (t < T) {
        const XT* xr = x + (size_t)t * H;
        float acc = 0.0f;
#pragma unroll 4
        for (int i = lane; i < H / 8; i += 32) {
            const int oa = (i >> 2) * 32 + (i & 3) * 4;
            const float4 p = x2f<XT>(xr + oa), q = x2f<XT>(xr + oa + 16);
            const float4 wp = __ldg(reinterpret_cast<const float4*>(w + oa)), wq = __ldg(reinterpret_cast<const float4*>(w + oa + 16));
            acc += p.x * wp.x + p.y * wp.y + p.z * wp.z + p.w * wp.w;
            acc += q.x * wq.x + q.y * wq.y + q.z * wq.z + q.w * wq.w;
            if (plane != nullptr) {
                auto pk = [](float a, float b) {
                    const __half2 h = __floats2half2_rn(a, b);
                    return *reinterpret_cast<const uint32_t*>(&h);
                };
                __half* dst = plane + (size_t)t * H;
                if (natural) {
                    *reinterpret_cast<uint2*>(dst + oa) = make_uint2(pk(p.x, p.y), pk(p.z, p.w));
                    *reinterpret_cast<uint2*>(dst + oa + 16) = make_uint2(pk(q.x, q.y), pk(q.z, q.w));
                } else {
                    reinterpret_cast<uint4*>(dst)[i] = make_uint4(pk(p.x, p.z), pk(q.x, q.z), pk(p.y, p.w), pk(q.y, q.w));
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) {
            float wt = 1.0f;  // gating 3
            if (gating == 2) {
                const float ex = lumen_exact::expf_libm_tab(-acc, lumen_exact::Exp2TabPtr{reinterpret_cast<const uint64_t*>(tab_s)});
                wt = __fdiv_rn(1.0f, __fadd_rn(1.0f, ex));
            }
            R.logits[t] = acc;
            R.ids[t] = 0u;
            R.weights[t] = wt;
            R.col_expert[t] = 0;
            R.col_src_tok[t] = t;
            R.dst_to_col[t] = t;
        }
    }
    if (blockIdx.x != 0) return;
    if (threadIdx.x == 0) {
        R.expert_bounds[0] = 0;
        R.expert_bounds[1] = T;
        R.uexp[0] = 0;
        *R.n_uexp = 1;
    }
#pragma unroll 1
    for (int which = 0; which < 2; ++which) {
        int4* tiles = which ? plan.tiles_dn : plan.tiles_gu;
        const int sh = which ? plan.tile_shift_dn : plan.tile_shift, mt_n = which ? plan.mt_dn : plan.mt_gu;
        const int n = ((T + (1 << sh) - 1) >> sh) * mt_n;
        for (int i = threadIdx.x; tiles != nullptr && i < n; i += 256) {
            const int c = i / mt_n;
            tiles[i] = make_int4(0, c << sh, min(1 << sh, T - (c << sh)), i - c * mt_n);
        }
        if (threadIdx.x == 0) plan.n_tiles[which] = n;
        if (threadIdx.x == 1) plan.n_tiles[2 + which] = 0;
    }
    if (plan.starts != nullptr) {
        const int n = (T + (1 << plan.tile_shift) - 1) >> plan.tile_shift;
        for (int i = threadIdx.x; i <= plan.ctas; i += 256) {
            plan.starts[i] = (int)((long long)n * plan.rt_gu * i / plan.ctas);
            plan.starts[plan.ctas + 1 + i] = (int)((long long)n * plan.rt_dn * i / plan.ctas);
        }
    }
}

bool route_single_applicable(const PrefillArgs& a) {
    return a.L.E == 1 && a.K == 1 && a.gating >= 2 && a.ids_in == nullptr && a.logits_override == nullptr && a.gamma == nullptr && a.act_dtype != 2 &&
           a.L.H % 32 == 0 && (reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.L.router_w)) % 16 == 0;
}

// One warp per chunk of SORT_TOK tokens: the chunk's (token, slot) pairs are taken 32 at
// a time in order; lanes holding the same expert find each other with match.any, the
// position inside the expert's segment is the expert's running cursor plus the number
// of lower lanes with the same expert, so the placement is stable.
// The segment bounds are a scan of the row totals, which every CTA does for itself, so that the plan (the last CTA) is made beside the
// placement and not in front of it. The rows of the histogram are read by expert, a lane per chunk (a warp reading its own
// chunk's column made as many requests as there are counts: 4096 tokens of 256 experts, top-k and sort 24.5 -> 20.8 us).
constexpr int PLACE_CHUNKS = PLAN_THREADS / 32;
__global__ void __launch_bounds__(PLAN_THREADS)
sort_place_kernel(const uint32_t* __restrict__ ids, int T, int K, const int32_t* __restrict__ blk_hist, int nchunks, RouteDev R,
                  const __grid_constant__ PlanArgs plan) {
    extern __shared__ int cursor[];  // [PLACE_CHUNKS][E | 1]
    __shared__ int cnt_s[MAX_EXPERTS], bounds_s[MAX_EXPERTS], wsum_s[MAX_EXPERTS / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, E = plan.E;
    grid_dep_sync();
    int x = 0, inc = 0;
    if (tid < MAX_EXPERTS) {
        x = (tid < E) ? blk_hist[(size_t)E * nchunks + tid] : 0;
        cnt_s[tid] = x;
    }
    if (blockIdx.x == gridDim.x - 1) {
        __syncthreads();
        emit_plan(plan, R, cnt_s, bounds_s);
        return;
    }
    if (tid < MAX_EXPERTS) {
        inc = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int w = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += w;
        }
        if (lane == 31) wsum_s[warp] = inc;
    }
    const int chunk0 = blockIdx.x * PLACE_CHUNKS, chunk = chunk0 + warp;
    int* cur = cursor + warp * (E | 1);  // (an odd stride: the lanes below hit 32 banks)
    if (chunk0 + lane < nchunks)
        for (int e = warp; e < E; e += PLACE_CHUNKS) cursor[lane * (E | 1) + e] = blk_hist[(size_t)e * nchunks + chunk0 + lane];
    __syncthreads();
    if (tid < MAX_EXPERTS) {
        int base = 0;
#pragma unroll
        for (int w = 0; w < MAX_EXPERTS / 32; ++w) base += (w < warp) ? wsum_s[w] : 0;
        bounds_s[tid] = base + inc - x;
    }
    __syncthreads();
    if (chunk >= nchunks) return;
    const int t0 = chunk * SORT_TOK;
    const int n = min(SORT_TOK, T - t0) * K;
    for (int p0 = 0; p0 < n; p0 += 32) {
        const int p = p0 + lane;
        const bool valid = p < n;
        const int e = valid ? (int)ids[(size_t)t0 * K + p] : -1 - lane;  // invalid lanes match nobody
        const unsigned int same = __match_any_sync(0xffffffffu, e);
        const int rank = __popc(same & ((1u << lane) - 1u));
        if (valid) {
            const int col = bounds_s[e] + cur[e] + rank;
            R.col_expert[col] = e;
            R.col_src_tok[col] = t0 + p / K;
            R.dst_to_col[(size_t)t0 * K + p] = col;
        }
        __syncwarp();
        if (valid && rank == 0) cur[e] += __popc(same);  // one leader per expert
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// activation fragments for the mma.sync grouped path (any T)
// ---------------------------------------------------------------------------
template <typename XT>
__global__ void __launch_bounds__(256)
build_xf_kernel(const XT* __restrict__ x, int T, int H, int nblk_pad, bool bf16_mode, uint4* __restrict__ xf) {
    const int nblk = H >> 5;
    const size_t idx = (size_t)blockIdx.x * 256 + threadIdx.x;
    const size_t total = (size_t)T * nblk * 8;
    if (idx >= total) return;
    const int sub = (int)(idx & 7), hl = sub >> 2, t4 = sub & 3;
    const size_t item = idx >> 3;
    const int t = (int)(item / nblk), b = (int)(item % nblk);
    const XT* xr = x + (size_t)t * H + b * 32;
    float4 lo4, hi4;
    lo4.x = x_to_f32<XT>(xr[4 * t4]);
    lo4.y = x_to_f32<XT>(xr[4 * t4 + 1]);
    lo4.z = x_to_f32<XT>(xr[4 * t4 + 2]);
    lo4.w = x_to_f32<XT>(xr[4 * t4 + 3]);
    hi4.x = x_to_f32<XT>(xr[16 + 4 * t4]);
    hi4.y = x_to_f32<XT>(xr[16 + 4 * t4 + 1]);
    hi4.z = x_to_f32<XT>(xr[16 + 4 * t4 + 2]);
    hi4.w = x_to_f32<XT>(xr[16 + 4 * t4 + 3]);
    xf[((size_t)(t * 2 + hl) * nblk_pad + b) * 4 + t4] = make_act_frag(lo4, hi4, hl, bf16_mode);
}

// ---------------------------------------------------------------------------
// scatter-accumulate
// ---------------------------------------------------------------------------
// One thread per 8 consecutive outputs (16-byte loads of the f16 rows); the slots are taken S
// at a time so that their rows are in flight together, and added in slot order: eight for a short batch, where the
// chain of round trips is the time (77 tokens: 6 -> 4 us), four when the rows come from HBM (4096 tokens: 33 us, 51
// with eight: fewer warps resident).
template <int S>  // slots in flight
__global__ void __launch_bounds__(256)
scatter_accum_kernel(const __half* __restrict__ d16, const float* residual,
                     const float* __restrict__ weights, const int32_t* __restrict__ dst_to_col,
                     float* out, int T, int H, int K) {  // residual may be out (in-place layer stacks)
    grid_dep_sync();
    const int t = blockIdx.x;  // tokens on grid.x: the y dimension is limited to 65535
    const int h8 = blockIdx.y * 256 + threadIdx.x;  // group of 8 outputs
    if (h8 * 8 >= H) return;
    const size_t o = (size_t)t * H + h8 * 8;
    float acc[8];
    {
        const float4 r0 = *reinterpret_cast<const float4*>(residual + o);
        const float4 r1 = *reinterpret_cast<const float4*>(residual + o + 4);
        acc[0] = r0.x; acc[1] = r0.y; acc[2] = r0.z; acc[3] = r0.w;
        acc[4] = r1.x; acc[5] = r1.y; acc[6] = r1.z; acc[7] = r1.w;
    }
    for (int s0 = 0; s0 < K; s0 += S) {
        int col[S];
        uint4 d[S];
        float w[S];
#pragma unroll
        for (int j = 0; j < S; ++j) {
            const size_t p = (size_t)t * K + min(s0 + j, K - 1);
            col[j] = dst_to_col[p];
            w[j] = weights[p];
        }
#pragma unroll
        for (int j = 0; j < S; ++j)
            if (s0 + j < K) d[j] = *reinterpret_cast<const uint4*>(d16 + (size_t)col[j] * H + h8 * 8);
#pragma unroll
        for (int j = 0; j < S; ++j) {
            if (s0 + j < K) {
                const __half2* hp = reinterpret_cast<const __half2*>(&d[j]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 f = __half22float2(hp[i]);
                    acc[2 * i] = __fadd_rn(acc[2 * i], __fmul_rn(w[j], f.x));
                    acc[2 * i + 1] = __fadd_rn(acc[2 * i + 1], __fmul_rn(w[j], f.y));
                }
            }
        }
    }
    *reinterpret_cast<float4*>(out + o) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    *reinterpret_cast<float4*>(out + o + 4) = make_float4(acc[4], acc[5], acc[6], acc[7]);
}

// The same, one output a thread, for what the 16-byte accesses above cannot take: rows that are no whole number of them
// (lumen_moe_combine_f16 takes any even hidden_dim) or a caller's buffer that lies between two such boundaries.
__global__ void __launch_bounds__(256)
scatter_accum_scalar_kernel(const __half* __restrict__ d16, const float* residual, const float* __restrict__ weights,
                            const int32_t* __restrict__ dst_to_col, float* out, int T, int H, int K) {
    grid_dep_sync();
    const int t = blockIdx.x, h = blockIdx.y * 256 + threadIdx.x;
    if (h >= H) return;
    float acc = residual[(size_t)t * H + h];
    for (int s = 0; s < K; ++s) {
        const size_t p = (size_t)t * K + s;
        acc = __fadd_rn(acc, __fmul_rn(weights[p], __half2float(d16[(size_t)dst_to_col[p] * H + h])));
    }
    out[(size_t)t * H + h] = acc;
}

cudaError_t launch_scatter_accum(const __half* d16, const float* residual, const RouteDev& R, float* out,
                                 int T, int H, int K, cudaStream_t st) {
    count_launch();
    const bool vec = H % 8 == 0 && (reinterpret_cast<uintptr_t>(d16) | reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(out)) % 16 == 0;
    if (!vec)
        return launch_dep(scatter_accum_scalar_kernel, dim3(T, (H + 255) / 256), dim3(256), 0, st, d16, residual, R.weights, R.dst_to_col, out,
                          T, H, K);
    return launch_dep(T <= 512 ? scatter_accum_kernel<8> : scatter_accum_kernel<4>, dim3(T, (H / 8 + 255) / 256), dim3(256), 0, st, d16, residual, R.weights,
                      R.dst_to_col, out, T, H, K);
}

__global__ void __launch_bounds__(256)
rows_from_cols_kernel(const __half* __restrict__ d16, const int32_t* __restrict__ dst_to_col, __half* __restrict__ out16,
                      int H) {
    const int t = blockIdx.x;
    const uint4* src = reinterpret_cast<const uint4*>(d16 + (size_t)dst_to_col[t] * H);
    uint4* dst = reinterpret_cast<uint4*>(out16 + (size_t)t * H);
    for (int i = threadIdx.x; i < H / 8; i += 256) dst[i] = src[i];
}

cudaError_t launch_rows_from_cols(const __half* d16, const int32_t* dst_to_col, __half* out16, int T, int H,
                                  cudaStream_t st) {
    count_launch();
    rows_from_cols_kernel<<<T, 256, 0, st>>>(d16, dst_to_col, out16, H);
    return cudaGetLastError();
}

cudaError_t launch_build_xf(const void* x, int act_dtype, int T, int H, int nblk_pad, bool bf16_mode,
                            uint4* xf, cudaStream_t st) {
    const size_t total = (size_t)T * (H / 32) * 8;
    count_launch();
    if (act_dtype == 0)
        build_xf_kernel<float><<<(unsigned)((total + 255) / 256), 256, 0, st>>>((const float*)x, T, H, nblk_pad,
                                                                               bf16_mode, xf);
    else if (act_dtype == 2)
        build_xf_kernel<__half><<<(unsigned)((total + 255) / 256), 256, 0, st>>>((const __half*)x, T, H, nblk_pad,
                                                                                bf16_mode, xf);
    else
        build_xf_kernel<__nv_bfloat16><<<(unsigned)((total + 255) / 256), 256, 0, st>>>(
            (const __nv_bfloat16*)x, T, H, nblk_pad, bf16_mode, xf);
    return cudaGetLastError();
}

// Caller-supplied routing (expert-parallel ranks receive rows that were routed
// elsewhere): copy the ids, weights default to 1. The reference checks expert_id < E on
// its host path (cuda/moe.rs:1776-1780); here the ids are device data, so the check runs
// on the device: an id >= E raises the context's status word (LUMEN_MOE_INVALID_ARG) and
// the pair is routed to expert 0 with weight 0, so that no table or histogram is ever
// indexed out of range.
__global__ void set_routing_kernel(const uint32_t* __restrict__ ids_in, const float* __restrict__ w_in, int n, int E,
                                   uint32_t* __restrict__ ids, float* __restrict__ w, int32_t* status,
                                   int32_t* status_host) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < n) {
        uint32_t id = ids_in[i];
        float wt = w_in ? w_in[i] : 1.0f;
        if (id >= (uint32_t)E) {
            if (status != nullptr) raise_status(status, status_host, 1);
            id = 0u;
            wt = 0.0f;
        }
        ids[i] = id;
        w[i] = wt;
    }
}

static int log2i(int v) { return v <= 1 ? 0 : 1 + log2i(v / 2); }

template <int NS>
static cudaError_t launch_topk_n(const PrefillArgs& a, const float* lg, int nparts, int32_t* hist, cudaStream_t st) {
    const dim3 grid((a.T + TK_WARPS - 1) / TK_WARPS), block(TK_WARPS * 32);
    auto go = [&](auto kern) {
        return launch_dep(kern, grid, block, 0, st, lg, a.R.logits, a.T, a.L.E, a.K, a.gating, a.R.ids, a.R.weights, hist);
    };
    switch (nparts) {
        case 0: return go(topk_large_kernel<NS, 0>);
        case 1: return go(topk_large_kernel<NS, 1>);
        case 2: return go(topk_large_kernel<NS, 2>);
        default: return go(topk_large_kernel<NS, 4>);
    }
}
static cudaError_t launch_topk(const PrefillArgs& a, const float* lg, int nparts, int32_t* hist, cudaStream_t st) {
    if (a.L.E <= 32) return launch_topk_n<1>(a, lg, nparts, hist, st);
    return (a.L.E <= 128) ? launch_topk_n<4>(a, lg, nparts, hist, st) : launch_topk_n<8>(a, lg, nparts, hist, st);
}

// Router + tables for any T. tile lists are optional (tiles == nullptr skips them).
cudaError_t launch_route_large(const PrefillArgs& a, cudaStream_t st) {
    const int T = a.T, E = a.L.E, H = a.L.H, K = a.K;
    const float* lg = a.logits_override;
    const int C = T * K;
    // columns per grouped-GEMM tile, the same for gate/up and down (the streaming kernels share one list of column chunks and cut the rows themselves)
    const bool stream = (a.impl == 2);
    const int tile_cols = stream ? STREAM_CHUNK : tc_form(a.L, C, a.sms, a.tc_ctas).cols, tile_cols_dn = tile_cols;
    const int max_ct = C / tile_cols + E, max_ct_dn = C / tile_cols_dn + E;
    const int mt_gu = stream ? 1 : a.L.I / 128, mt_dn = a.L.H / 256;  // m-tiles: 128 gate + 128 up rows | 256 down rows
    int4* tiles_gu = a.tiles;
    int4* tiles_dn = (a.tiles && !stream) ? a.tiles + (size_t)max_ct * (mt_gu > 0 ? mt_gu : 1) : nullptr;
    const PlanArgs plan{E, log2i(tile_cols), log2i(tile_cols_dn), mt_gu, mt_dn, tiles_gu, tiles_dn, a.n_tiles, max_ct * mt_gu, max_ct_dn * mt_dn,
                        a.any_lo, stream ? a.stream_starts : nullptr, a.sms, a.L.I / 16, a.L.H / 16};
    if (route_single_applicable(a)) {
        count_launch();
        __half* plane = (a.impl != 1) ? a.xr16 : nullptr;
        const bool natural = a.L.planes_natural && !stream;
        const dim3 grid((T + 7) / 8), block(256);
        if (a.act_dtype == 0)
            return launch_dep(route_single_kernel<float>, grid, block, 0, st, (const float*)a.x, a.L.router_w, T, H, a.gating, a.R, plane, natural, plan);
        return launch_dep(route_single_kernel<__nv_bfloat16>, grid, block, 0, st, (const __nv_bfloat16*)a.x, a.L.router_w, T, H, a.gating, a.R,
                          plane, natural, plan);
    }
    int nparts = 0;
    if (a.ids_in != nullptr) {
        count_launch();
        set_routing_kernel<<<(T * K + 255) / 256, 256, 0, st>>>(a.ids_in, a.weights_in, T * K, E, a.R.ids, a.R.weights,
                                                                a.status, a.status_host);
    } else if (lg == nullptr && a.L.router_w16 != nullptr && a.xr16 != nullptr && a.rpart != nullptr &&
               router_tc_applicable(T, E, H, a.x)) {
        // tcgen05 router: partial logits per k range, summed by the top-k kernel
        nparts = router_tc_ksplit(H);
        if (a.gamma != nullptr)
            CUDA_RET(launch_norm_split(static_cast<const float*>(a.x), a.gamma, a.eps, T, H, a.L.planes_natural, a.xr16, a.any_lo, st));
        else
            CUDA_RET(launch_split_x16(a.x, a.act_dtype, T, H, a.L.planes_natural, a.xr16, a.any_lo, st));
        CUDA_RET(launch_router_logits_tc(a.L.router_w16, T, E, H, nparts, a.sms, a.xr16, a.any_lo, a.rpart, a.status, a.status_host,
                                         a.wait_limit_us, st));
        lg = a.rpart;
    } else if (lg == nullptr) {
        count_launch();
        if (H % 32 == 0 && a.w16 != nullptr && reinterpret_cast<uintptr_t>(a.x) % 16 == 0) {
            const size_t n = (size_t)E * H;
            split_router_w_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(a.L.router_w, a.w16, n);
            count_launch(1);
            // experts per CTA: fewer for small batches, so that every SM still gets several warps
            const int ne = (T <= 2048) ? 16 : (T <= 16384) ? 32 : 64;
            const dim3 grid((T + 63) / 64, (E + ne - 1) / ne);
#define LUMEN_LAUNCH_LOGITS(XT, NE_) \
    router_logits_mma_kernel<XT, NE_><<<grid, 128, 0, st>>>((const XT*)a.x, a.w16, a.R.logits, T, H, E)
            if (a.act_dtype == 0) {
                if (ne == 16) LUMEN_LAUNCH_LOGITS(float, 16);
                else if (ne == 32) LUMEN_LAUNCH_LOGITS(float, 32);
                else LUMEN_LAUNCH_LOGITS(float, 64);
            } else {
                if (ne == 16) LUMEN_LAUNCH_LOGITS(__nv_bfloat16, 16);
                else if (ne == 32) LUMEN_LAUNCH_LOGITS(__nv_bfloat16, 32);
                else LUMEN_LAUNCH_LOGITS(__nv_bfloat16, 64);
            }
#undef LUMEN_LAUNCH_LOGITS
        } else {
            const dim3 grid((T + 63) / 64, (E + 63) / 64);
            if (a.act_dtype == 0)
                router_logits_large_kernel<float><<<grid, 256, 0, st>>>((const float*)a.x, a.L.router_w, a.R.logits, T, H, E);
            else
                router_logits_large_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>((const __nv_bfloat16*)a.x, a.L.router_w,
                                                                               a.R.logits, T, H, E);
        }
        lg = a.R.logits;
    }
    const int nchunks = (T + SORT_TOK - 1) / SORT_TOK;
    const bool one_cta = T * K <= SORT1_MAX;
    count_launch(one_cta ? 2 : 3);
    if (a.ids_in == nullptr)
        CUDA_RET(launch_topk(a, lg, nparts, one_cta ? nullptr : a.blk_hist, st));
    else if (!one_cta)
        CUDA_RET(launch_dep(sort_hist_kernel, dim3(nchunks), dim3(256), 0, st, a.R.ids, T, K, E, a.blk_hist));
    if (one_cta) return launch_dep(sort_one_kernel, dim3(1), dim3(SORT1_WARPS * 32), 0, st, a.R.ids, C, K, a.R, plan);
    CUDA_RET(launch_dep(sort_rowscan_kernel, dim3(E), dim3(32), 0, st, a.blk_hist, nchunks));
    return launch_dep(sort_place_kernel, dim3((nchunks + PLACE_CHUNKS - 1) / PLACE_CHUNKS + 1), dim3(PLAN_THREADS), (size_t)PLACE_CHUNKS * (E | 1) * 4, st, a.R.ids, T,
                      K, a.blk_hist, nchunks, a.R, plan);
}

cudaError_t launch_tile_plan(const RouteDev& R, int E, int H, int I, int rows_cap, int gu_cols, int4* tiles,
                             int32_t* n_tiles, cudaStream_t st, const int32_t* stream_mode, int4* chunks, int32_t* starts,
                             int sms) {
    const int max_ct = rows_cap / gu_cols + E, max_ct_dn = rows_cap / 128 + E;
    const int mt_gu = I / 128, mt_dn = H / 256;
    count_launch();
    // (down tiles of 128 tokens here: an expert-parallel down product stores its rows into other GPUs'
    // memory, which only the always-overlapped epilogue of the 128-token form hides)
    const PlanArgs plan{E, log2i(gu_cols), 7, mt_gu, mt_dn, tiles, tiles + (size_t)max_ct * (mt_gu > 0 ? mt_gu : 1), n_tiles,
                        max_ct * mt_gu, max_ct_dn * mt_dn, nullptr, stream_mode ? starts : nullptr, sms, I / 16, H / 16,
                        stream_mode, chunks};
    return launch_dep(sort_scan_kernel, dim3(1), dim3(PLAN_THREADS), 0, st, plan, R);
}

// ---------------------------------------------------------------------------
// Expert-parallel send side in one launch: activation rows gathered in compact-column
// order (= destination-rank order, experts being contiguous per rank) as bf16, the
// expert id of every row relative to its rank, and the number of rows per rank.
// ---------------------------------------------------------------------------
// XT = float: rows leave as f16 (round to nearest, what the grouped GEMM's gather applies to
// f32 activations); XT = bf16: rows leave as bf16, unchanged.
template <typename XT>
__global__ void __launch_bounds__(256)
ep_prepare_kernel(const XT* __restrict__ x, RouteDev R, int H, int E, int epr, uint16_t* __restrict__ rows,
                  int32_t* __restrict__ local_ids, long long* __restrict__ send_counts) {
    const int col = blockIdx.x;
    const int tok = R.col_src_tok[col];
    const XT* src = x + (size_t)tok * H;
    uint16_t* dst = rows + (size_t)col * H;
    for (int i = threadIdx.x * 8; i < H; i += 256 * 8) {
        __align__(16) uint16_t v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (sizeof(XT) == 4) v[j] = __half_as_ushort(__float2half_rn(x_to_f32<XT>(src[i + j])));
            else v[j] = reinterpret_cast<const uint16_t*>(src)[i + j];
        }
        *reinterpret_cast<uint4*>(dst + i) = *reinterpret_cast<const uint4*>(v);
    }
    if (threadIdx.x == 0) local_ids[col] = R.col_expert[col] % epr;
    if (col == 0) {
        for (int r = threadIdx.x; r * epr < E; r += 256)
            send_counts[r] = (long long)(R.expert_bounds[min((r + 1) * epr, E)] - R.expert_bounds[r * epr]);
    }
}

cudaError_t launch_ep_prepare(const void* x, int act_dtype, const RouteDev& R, int C, int H, int E, int epr, void* rows,
                              int32_t* local_ids, long long* send_counts, cudaStream_t st) {
    count_launch();
    if (act_dtype == 0)
        ep_prepare_kernel<float><<<C, 256, 0, st>>>((const float*)x, R, H, E, epr, (uint16_t*)rows, local_ids, send_counts);
    else
        ep_prepare_kernel<__nv_bfloat16><<<C, 256, 0, st>>>((const __nv_bfloat16*)x, R, H, E, epr, (uint16_t*)rows,
                                                            local_ids, send_counts);
    return cudaGetLastError();
}

}  // namespace lumen
