// Router logits of a multi-token batch on the 5th-generation tensor cores:
//   logit[t, e] = sum_j W_r[e, j] * x[t, j]        (moe_router_logits_batched,
//                                                   cuda/shaders/moe_grouped.cu:79; CPU: cuda/moe.rs:6456-6463)
// with f32-grade accuracy from 16-bit operands: W_r and x are each split into a high and a
// low f16 part (w = w_hi + w_lo to ~2^-22 relative) and the three products w_hi x_hi +
// w_lo x_hi + w_hi x_lo accumulate in ONE f32 accumulator in TMEM (the dropped w_lo x_lo term is
// ~2^-22 relative). The x_lo product is skipped for a batch whose low parts are all zero
// (bf16 activations).
//
// Formulation: the router weight is the M operand (128 expert rows per tile, E <= 256 ->
// one or two row tiles), tokens are the N columns (128 per tile), and the contraction is cut
// into `ksplit` ranges so that a few thousand tokens still fill the machine: CTA (token tile,
// row tile, k range) writes its partial logits, and the top-k kernel adds the ksplit partials
// in a fixed order (deterministic, no atomics). Everything is fed by TMA: the f16 planes of
// W_r are built once per layer, those of x by a pre-pass over the batch.
//
//   thread 0 of warp 0   TMA producer (4 boxes of 64 inputs per stage: W_hi, W_lo, x_hi, x_lo)
//   thread 0 of warp 1   tcgen05.mma issue, tcgen05.commit frees the stages
//   warps 2..5           epilogue: tcgen05.ld, coalesced f32 stores (lane = expert)
// All mbarrier waits are bounded; on expiry the kernel raises the context's status word,
// frees its TMEM and returns.
#include "tc_common.cuh"
#include <type_traits>

namespace lumen {

namespace rtc {

using namespace tc;

// Tokens per tile: 32, 64, 128 or 256, whichever moves the fewest bytes through its waves of CTAs (every tile reads the weight
// planes of its k range). A logit is the same in all of them: the tile width only says how many columns one MMA covers.
// (77 tokens: 11 us with 128, 6 with 32, the set-up and the first weight boxes ahead of the wait for the kernel before.)
template <int BN>
struct Cfg {
    static constexpr int STAGES = (BN == 256) ? 2 : (BN == 128) ? 3 : (BN == 64) ? 4 : 5;
    static constexpr int X_BYTES = BN * 128;                           // [BN rows x 64 k] f16
    static constexpr int STAGE_BYTES = 2 * SUB_BYTES + 2 * X_BYTES;    // W_hi | W_lo ([128 rows x 64 k] each) | x_hi | x_lo
};
constexpr int THREADS = 6 * 32;

struct Args {
    CUtensorMap tmap_w;   // [2 E, H] f16: rows [0, E) high parts, [E, 2 E) low parts
    CUtensorMap tmap_x;   // [2 T, H] f16: rows [0, T) high parts, [T, 2 T) low parts
    float* part;          // [ksplit][T][E] partial logits
    const int32_t* any_lo;  // non-zero when some low part of x is non-zero
    int32_t* status;
    int32_t* status_host;
    uint64_t wait_limit_ns;
    int T, E, H, ksplit, m_tiles;
};

template <int BN>
__global__ void __launch_bounds__(THREADS, 1)
router_logits_tc_kernel(const __grid_constant__ Args a) {
    constexpr int STAGES = Cfg<BN>::STAGES, STAGE_BYTES = Cfg<BN>::STAGE_BYTES, X_BYTES = Cfg<BN>::X_BYTES;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], acc_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ uint32_t abort_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t stage0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const AbortCtl abort_flag{&abort_s, a.wait_limit_ns};

    // tile of this CTA
    int idx = blockIdx.x;
    const int ks = idx % a.ksplit;
    idx /= a.ksplit;
    const int mt = idx % a.m_tiles;
    const int tt = idx / a.m_tiles;
    const int t0 = tt * BN, e0 = mt * 128;
    const int kh_per = (a.H / 64) / a.ksplit;  // 64-input stages of this CTA's k range
    const int kh0 = ks * kh_per;
    if (tid == 0) {
        abort_s = 0u;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 2);  // the weight boxes' and the activation boxes' expect_tx
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        mbar_init(smem_u32(&acc_bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                     "r"((uint32_t)BN)  // (a power of two, 32 at least)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;

    // The weight planes are static: their boxes of the first stages are requested before the wait for the split
    // kernel, whose output (the planes of x and the flag) everything else here depends on.
    auto load_w = [&](int n) {
        const int s = n % STAGES, k = (kh0 + n) * 64;
        const uint32_t bar = smem_u32(&full_bar[s]), base = stage0 + s * STAGE_BYTES;
        mbar_expect_tx(bar, 2 * SUB_BYTES);
        tma_load_2d(base, &a.tmap_w, k, e0, bar);
        tma_load_2d(base + SUB_BYTES, &a.tmap_w, k, a.E + e0, bar);
    };
    if (tid == 0)
        for (int n = 0; n < STAGES && n < kh_per; ++n) load_w(n);
    grid_dep_sync();
    const bool use_lo = (*a.any_lo != 0);

    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            int n = 0;
            for (; ok && n < kh_per; ++n) {
                const int s = n % STAGES, ph = (n / STAGES) & 1;
                if (n >= STAGES) {
                    ok = mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1, abort_flag);
                    if (!ok) break;
                    load_w(n);
                }
                const uint32_t bar = smem_u32(&full_bar[s]), base = stage0 + s * STAGE_BYTES + 2 * SUB_BYTES;
                const int k = (kh0 + n) * 64;
                mbar_expect_tx(bar, (use_lo ? 2 : 1) * X_BYTES);
                tma_load_2d(base, &a.tmap_x, k, t0, bar);
                if (use_lo) tma_load_2d(base + X_BYTES, &a.tmap_x, k, a.T + t0, bar);
            }
            if (!ok) let_land(smem_u32(&full_bar[0]), STAGES, n);
        }
        __syncwarp();
    } else if (warp == 1) {
        const uint32_t idesc = make_idesc(BN, false);
        bool ok = true;
        for (int n = 0, s = 0, ph = 0; n < kh_per; ++n) {
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&full_bar[s]), ph, abort_flag));
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint64_t w0 = make_desc(stage0 + s * STAGE_BYTES), x0 = w0 + (2 * SUB_BYTES >> 4);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    umma(tmem_base, w0 + j * 2, x0 + j * 2, idesc, (n > 0 || j > 0) ? 1u : 0u);
                    umma(tmem_base, w0 + (SUB_BYTES >> 4) + j * 2, x0 + j * 2, idesc, 1u);
                    if (use_lo) umma(tmem_base, w0 + j * 2, x0 + (X_BYTES >> 4) + j * 2, idesc, 1u);
                }
                umma_commit(smem_u32(&empty_bar[s]));
                if (n == kh_per - 1) umma_commit(smem_u32(&acc_bar));
            }
            __syncwarp();
            if (++s == STAGES) {
                s = 0;
                ph ^= 1;
            }
        }
    } else {
        // epilogue: warp w reads TMEM lanes 32 * (w % 4) ..; lane = expert row of the tile
        const int q = warp & 3;
        const int e = e0 + q * 32 + lane;
        if (mbar_wait(smem_u32(&acc_bar), 0, abort_flag)) {
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16);
            float* dst = a.part + ((size_t)ks * a.T + t0) * a.E + e;
            for (int n0 = 0; n0 < BN && t0 + n0 < a.T; n0 += 16) {
                uint32_t v[16];
                tmem_ld16(taddr + n0, v);
                tmem_ld_wait();
                if (e < a.E) {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (t0 + n0 + j < a.T) dst[(size_t)(n0 + j) * a.E] = __uint_as_float(v[j]);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)BN) : "memory");
    }
    if (tid == 0 && abort_s) raise_status(a.status, a.status_host, 4);  // LUMEN_MOE_TIMEOUT
}

// x [T, H] (f32, bf16 or f16) -> f16 planes [2][T][H] in the element order of the router weight's planes: high
// part, low part; *any_lo |= (some low part != 0). The high plane is also the activation operand of the expert
// products. any_lo null: no low plane wanted (routing supplied by the caller).
//
// Element order. Permuted (layers whose weights are dequantised): the order the dequantiser emits, 16-byte chunk t of a
// 32-block holding inputs (4t, 4t+2, 16+4t, 16+4t+2, 4t+1, 4t+3, 16+4t+1, 16+4t+3). Natural (weights copied by
// TMA from plain f16 matrices). A thread has inputs 4t.. (p) and 16+4t.. (q) of chunk i = 4 * block + t in both.
struct PlaneOut {
    __half* out;      // high plane, the low one `plane` elements on
    size_t plane;
    int32_t* any_lo;  // or null
    bool natural;
};
__device__ __forceinline__ unsigned store_planes(const PlaneOut& o, size_t i, const float4& p, const float4& q) {
    unsigned nz = 0u;
    const float f[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
    uint32_t hi[8], lo[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const __half h = __float2half_rn(f[j]);
        const __half l = __float2half_rn(f[j] - __half2float(h));
        hi[j] = __half_as_ushort(h);
        lo[j] = __half_as_ushort(l);
        nz |= lo[j] & 0x7fffu;
    }
    auto pair = [](const uint32_t (&v)[8], int a, int b) { return v[a] | (v[b] << 16); };
#pragma unroll
    for (int pl = 0; pl < 2; ++pl) {
        if (pl == 1 && o.any_lo == nullptr) break;
        const uint32_t(&v)[8] = pl ? lo : hi;
        __half* dst = o.out + (pl ? o.plane : 0);
        if (o.natural) {
            const size_t oa = (i >> 2) * 32 + (i & 3) * 4;
            *reinterpret_cast<uint2*>(dst + oa) = make_uint2(pair(v, 0, 1), pair(v, 2, 3));
            *reinterpret_cast<uint2*>(dst + oa + 16) = make_uint2(pair(v, 4, 5), pair(v, 6, 7));
        } else {
            reinterpret_cast<uint4*>(dst)[i] = make_uint4(pair(v, 0, 2), pair(v, 4, 6), pair(v, 1, 3), pair(v, 5, 7));
        }
    }
    return nz;
}
__device__ __forceinline__ void note_low_parts(const PlaneOut& o, unsigned nz) {
    // one warp's finding is enough: the word is read first, so that thousands of atomics do not queue on it
    if (o.any_lo != nullptr && __any_sync(0xffffffffu, nz != 0u) && (threadIdx.x & 31) == 0 &&
        *reinterpret_cast<volatile int32_t*>(o.any_lo) == 0)
        atomicOr(o.any_lo, 1);
}

template <typename XT>
__global__ void __launch_bounds__(256)
split_x16_kernel(const XT* __restrict__ x, size_t n8, const PlaneOut o) {
    grid_dep_sync();
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    unsigned nz = 0u;
    if (i < n8) {
        const size_t oa = (i >> 2) * 32 + (i & 3) * 4;
        float4 p, q;  // inputs 4t.. and 16+4t..
        if (sizeof(XT) == 4) {
            p = *reinterpret_cast<const float4*>(x + oa);
            q = *reinterpret_cast<const float4*>(x + oa + 16);
        } else {
            const uint2 u = *reinterpret_cast<const uint2*>(x + oa), v = *reinterpret_cast<const uint2*>(x + oa + 16);
            if (std::is_same<XT, __half>::value) {
                const float2 u0 = __half22float2(*reinterpret_cast<const __half2*>(&u.x)), u1 = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
                const float2 v0 = __half22float2(*reinterpret_cast<const __half2*>(&v.x)), v1 = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
                p = make_float4(u0.x, u0.y, u1.x, u1.y);
                q = make_float4(v0.x, v0.y, v1.x, v1.y);
            } else {
                p = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                                __uint_as_float(u.y & 0xffff0000u));
                q = make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                                __uint_as_float(v.y & 0xffff0000u));
            }
        }
        nz = store_planes(o, i, p, q);
    }
    note_low_parts(o, nz);
}

// RMSNorm (cuda/shaders/norm.cu:28-76) and the planes of its result in one pass over a layer stack's residual stream: one
// CTA per row, the row held in registers (H <= 8192). The squares are summed in the order of rmsnorm_kernel. At 8192
// tokens, H = 2048: 72 us as two kernels with the f32 result in between, 26 us (bytes: 128 MB, 20 us at the copy peak).
constexpr int NORM_MAX_CHUNKS = 4;
template <int NCH, int ROWS>  // NCH * 2048 >= H
__global__ void __launch_bounds__(256)
norm_split_kernel(const float* __restrict__ x, const float* __restrict__ gamma, float eps, int T, int H, const PlaneOut o) {
    grid_dep_sync();
    __shared__ float red[ROWS][8];
    const int t0 = blockIdx.x * ROWS, tid = threadIdx.x, n8 = H >> 3;
    float4 p[ROWS][NCH], q[ROWS][NCH];
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int j = 0; j < NCH; ++j) {
            const int i = tid + j * 256;
            if (i < n8) {
                const float* xr = x + (size_t)min(t0 + r, T - 1) * H + (i >> 2) * 32 + (i & 3) * 4;
                p[r][j] = *reinterpret_cast<const float4*>(xr);
                q[r][j] = *reinterpret_cast<const float4*>(xr + 16);
            }
        }
    float sc[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        float ss = 0.0f;
#pragma unroll
        for (int j = 0; j < NCH; ++j)
            if (tid + j * 256 < n8) ss = norm_sq_chunk(ss, p[r][j], q[r][j]);
        sc[r] = norm_scale(ss, red[r], H, eps);
    }
    unsigned nz = 0u;
#pragma unroll
    for (int j = 0; j < NCH; ++j) {
        const int i = tid + j * 256;
        if (i < n8) {
            const int oa = (i >> 2) * 32 + (i & 3) * 4;
            const float4 g = __ldg(reinterpret_cast<const float4*>(gamma + oa)), h = __ldg(reinterpret_cast<const float4*>(gamma + oa + 16));
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                // (rounded products: contracted into the subtraction of the high part they would not be the norm's outputs)
                auto normed = [&](const float4& v, const float4& w) {
                    return make_float4(__fmul_rn(__fmul_rn(v.x, sc[r]), w.x), __fmul_rn(__fmul_rn(v.y, sc[r]), w.y),
                                       __fmul_rn(__fmul_rn(v.z, sc[r]), w.z), __fmul_rn(__fmul_rn(v.w, sc[r]), w.w));
                };
                const float4 np = normed(p[r][j], g), nq = normed(q[r][j], h);
                if (t0 + r < T) nz |= store_planes(o, (size_t)(t0 + r) * n8 + i, np, nq);
            }
        }
    }
    note_low_parts(o, nz);
}

}  // namespace rtc

// W_r [E, H] f32 -> f16 planes [2][E][H] (high, low) in the same element order as x: once per layer
__global__ void split_router_w16_kernel(const float* __restrict__ w, __half* __restrict__ w16, size_t n, bool natural) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v = w[i];
    const __half hi = __float2half_rn(v);
    const int el = (int)(i & 31), t = (el & 15) >> 2, m = el & 3;
    const size_t o = natural ? i : (i & ~(size_t)31) + t * 8 + ((m & 1) ? 4 : 0) + ((el >> 4) ? 2 : 0) + (m >> 1);
    w16[o] = hi;
    w16[n + o] = __float2half_rn(v - __half2float(hi));
}

cudaError_t launch_split_router_w16(const float* w, __half* w16, int E, int H, bool natural, cudaStream_t st) {
    const size_t n = (size_t)E * H;
    count_launch();
    split_router_w16_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(w, w16, n, natural);
    return cudaGetLastError();
}

// k ranges per tile: a function of the shape only, never of the batch size, so that a token's
// logits (the order in which its partial sums are added) do not depend on how many tokens it is
// routed with: an expert-parallel rank routing its shard must get the bits one GPU gets for the
// whole batch. Four ranges of whole 64-input stages when H allows (a few thousand tokens then
// fill the machine), else two, else one.
int router_tc_ksplit(int H) {
    const int stages = H / 64;
    return (stages % 4 == 0) ? 4 : (stages % 2 == 0) ? 2 : 1;
}

bool router_tc_applicable(int T, int E, int H, const void* x) {
    return H % 64 == 0 && E >= 1 && E <= 256 && T >= 1 && reinterpret_cast<uintptr_t>(x) % 16 == 0;
}

cudaError_t launch_split_x16(const void* x, int act_dtype, int T, int H, bool natural, __half* x16, int32_t* any_lo, cudaStream_t st) {
    const size_t n8 = (size_t)T * H / 8;
    const rtc::PlaneOut o{x16, (size_t)T * H, any_lo, natural};
    const dim3 grid((unsigned)((n8 + 255) / 256));
    count_launch();
    if (act_dtype == 0) return launch_dep(rtc::split_x16_kernel<float>, grid, dim3(256), 0, st, (const float*)x, n8, o);
    if (act_dtype == 2) return launch_dep(rtc::split_x16_kernel<__half>, grid, dim3(256), 0, st, (const __half*)x, n8, o);
    return launch_dep(rtc::split_x16_kernel<__nv_bfloat16>, grid, dim3(256), 0, st, (const __nv_bfloat16*)x, n8, o);
}

bool norm_split_applicable(int H, const void* x, const void* gamma) {
    return H % 32 == 0 && H <= rtc::NORM_MAX_CHUNKS * 2048 && (reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gamma)) % 16 == 0;
}

cudaError_t launch_norm_split(const float* x, const float* gamma, float eps, int T, int H, bool natural, __half* x16, int32_t* any_lo,
                              cudaStream_t st) {
    const rtc::PlaneOut o{x16, (size_t)T * H, any_lo, natural};
    count_launch();
    // (two rows a CTA where the batch fills the chip: twice the loads in flight)
    const int rows = (H <= 2048 && T >= 4096) ? 2 : 1;
    auto kern = rows == 2 ? rtc::norm_split_kernel<1, 2>
                : H <= 2048 ? rtc::norm_split_kernel<1, 1>
                : H <= 4096 ? rtc::norm_split_kernel<2, 1>
                            : rtc::norm_split_kernel<rtc::NORM_MAX_CHUNKS, 1>;
    return launch_dep(kern, dim3((T + rows - 1) / rows), dim3(256), 0, st, x, gamma, eps, T, H, o);
}

template <int BN>
static cudaError_t launch_rtc(const rtc::Args& a, cudaStream_t st) {
    const int smem = rtc::Cfg<BN>::STAGES * rtc::Cfg<BN>::STAGE_BYTES + 1024;
    static SmemOptIn optin;
    const cudaError_t e = ensure_dyn_smem(rtc::router_logits_tc_kernel<BN>, (size_t)smem, optin);
    if (e != cudaSuccess) return e;
    const int grid = ((a.T + BN - 1) / BN) * a.m_tiles * a.ksplit;
    return launch_dep(rtc::router_logits_tc_kernel<BN>, dim3(grid), dim3(rtc::THREADS), (size_t)smem, st, a);
}

// logits partials of the whole batch from its planes (launch_split_x16 or launch_norm_split); part is scratch of the context
cudaError_t launch_router_logits_tc(const __half* w16, int T, int E, int H, int ksplit, int sms,
                                    const __half* x16, int32_t* any_lo, float* part, int32_t* status, int32_t* status_host,
                                    unsigned wait_limit_us, cudaStream_t st) {
    count_launch();
    rtc::Args a{};
    a.m_tiles = (E + 127) / 128;
    cudaError_t e = make_tmap_f16(w16, (uint64_t)2 * E, (uint64_t)H, 128, &a.tmap_w);
    if (e != cudaSuccess) return e;
    // The least bytes of a CTA's stage (weights + activations) times the waves of CTAs. Two measured exceptions: tiles of 64 tokens lose to
    // half as many of 128 from 5/7 of the SMs on, and tiles of 256 to a second wave of 128 that is short (the whole routing, us, f32 and bf16-valued rows,
    // H = 2048, by tile width. E = 128: 1200 tokens 32 39.7 and 29.5, 64 37.2 and 26.6; 1800 tokens 32 46.5 and 33.4, 64 (116 CTAs) 47.5 and 35.3, 128 46.6
    // and 29.9; 8192 tokens 128 87.7 and 68.3, 256 84.5 and 65.3. E = 256: 832 tokens 64 (104 CTAs) 37.7 and 29.4, 128 39.7 and 30.6; 896 tokens 64 (112)
    // 44.2 and 36.3, 128 39.6 and 31.7; 2500 tokens 128 (160) 60.3 and 45.7, 256 67.2 and 49.3; 3000 tokens 128 (192) 66.8 and 52.3, 256 64.4 and 49.5)
    int bn = 32;
    long long least = 0, before = 0;  // before: CTAs of the width before
    for (int b = 32; b <= 256; b *= 2) {
        const long long ctas = (long long)((T + b - 1) / b) * a.m_tiles * ksplit, room = b == 64 ? sms * 5 / 7 : sms;
        const long long cost = (ctas + room - 1) / room * (2 * tc::SUB_BYTES + 2 * b * 128);
        if (b == 32 || (cost <= least && !(b == 256 && 4 * before < 5 * sms))) {
            least = cost;
            bn = b;
        }
        before = ctas;
    }
    e = make_tmap_f16(x16, (uint64_t)2 * T, (uint64_t)H, bn, &a.tmap_x);
    if (e != cudaSuccess) return e;
    a.part = part;
    a.any_lo = any_lo;
    a.status = status;
    a.status_host = status_host;
    a.wait_limit_ns = wait_limit_us ? (uint64_t)wait_limit_us * 1000ull : tc::WAIT_LIMIT_NS;
    a.T = T;
    a.E = E;
    a.H = H;
    a.ksplit = ksplit;
    return bn == 32 ? launch_rtc<32>(a, st) : bn == 64 ? launch_rtc<64>(a, st) : bn == 128 ? launch_rtc<128>(a, st) : launch_rtc<256>(a, st);
}

}  // namespace lumen
