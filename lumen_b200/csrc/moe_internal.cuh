// Internal declarations shared by the kernels and the host layer of the MoE
// operator: device-side layouts, scratch buffers and launch prototypes.
#pragma once
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <stddef.h>

namespace lumen {

enum Quant : int { Q8_0 = 0, Q4_0 = 1, BF16 = 2 };

constexpr int MAX_EXPERTS = 256;  // cuda/shaders/moe_router.cu:33
constexpr int MAX_TOP_K = 16;     // cuda/shaders/moe_router.cu:34
constexpr int DECODE_MAX_TOKENS = 16;

// ---------------------------------------------------------------------------
// Repacked expert weights ("fragment planes").
//
// A matrix [R rows, Kdim] (rows = outputs, Kdim = inputs, 32-element blocks along
// Kdim) is cut into tiles of 16 rows x 4 blocks (128 inputs). Tile (rt, kg) is
// stored as NQ consecutive 512-byte vectors (one uint4 per lane of a warp), laid
// out so that lane (g = lane/4, t = lane%4) finds in its own uint4s exactly the
// words the m16n8k16 A fragment of rows {16rt+g, 16rt+g+8} needs:
//   Q4_0 (NQ=2): vector j holds blocks 2j, 2j+1 of the group:
//        {w(g,2j,t), w(g+8,2j,t), w(g,2j+1,t), w(g+8,2j+1,t)}, w(r,b,t) = 32-bit
//        word t of the block's 16 nibble bytes (elements 4t..4t+3 low nibbles,
//        16+4t..16+4t+3 high nibbles).
//   Q8_0 (NQ=4): vector b holds block b: {w(g,b,t), w(g,b,4+t), w(g+8,b,t), w(g+8,b,4+t)},
//        w(r,b,i) = 32-bit word i of the block's 32 int8 (elements 4i..4i+3).
//   BF16 (NQ=8): vector 2b+r holds, for row g+8r, the 8 bf16 elements
//        {4t..4t+3, 16+4t..16+4t+3} of block b.
// Scales (Q4_0/Q8_0): per tile 8 uint4, one per g: f16 {row g: blocks 0..3, row g+8: blocks 0..3}.
// Blocks past Kdim inside the last group are zero (scale 0).
// ---------------------------------------------------------------------------
struct LayerDev {
    const uint8_t* blob;
    const float* router_w;  // blob + router_off, [E,H] f32
    const __half* router_w16;  // [2][E][H] f16 high / low parts of router_w (batched router on tcgen05), or null
    bool planes_natural;       // element order of these planes and of the activations' (see route_tc.cu)
    const uint4* q;         // all experts' quant planes
    const uint4* s;         // all experts' scale planes (unused for BF16)
    // optional plain f16 matrices of all experts (scale folded in) for the TMA-fed prefill products:
    // gu16 [E][2 I rows: gate then up][H], dn16 [E][H rows][I]; null = dequantise in shared memory
    const __half* gu16;
    const __half* dn16;
    int quant, H, I, E;
    int kg_h, kg_i;  // 128-input groups along H (gate/up) and I (down)
    int rt_i, rt_h;  // 16-row tiles of gate/up (I rows) and down (H rows)
    int nq;          // uint4 per lane per tile
    size_t q_gu, q_dn, q_exp;  // uint4 counts: one gate (or up) matrix, one down matrix, one expert
    size_t s_gu, s_dn, s_exp;

    __host__ __device__ const uint4* gate_q(int e) const { return q + (size_t)e * q_exp; }
    __host__ __device__ const uint4* up_q(int e) const { return q + (size_t)e * q_exp + q_gu; }
    __host__ __device__ const uint4* down_q(int e) const { return q + (size_t)e * q_exp + 2 * q_gu; }
    __host__ __device__ const uint4* gate_s(int e) const { return s + (size_t)e * s_exp; }
    __host__ __device__ const uint4* up_s(int e) const { return s + (size_t)e * s_exp + s_gu; }
    __host__ __device__ const uint4* down_s(int e) const { return s + (size_t)e * s_exp + 2 * s_gu; }
};

// Form of the tcgen05 products of a one-GPU call: columns per tile, and whether CTA pairs work them (prefill_pair.cu: 512 or
// 128 columns) or single CTAs (prefill_tc.cu, only where the grid is capped at one: 256 or 128).
// Pairs, 512: once the experts average so many columns that tiles of 128 would be cut often (E = 128, I = 768, us from the host, tiles of
// 128 and of 512: Q4_0 112 columns 249 and 261, 128 columns 301 and 275; f16 matrices, whose weights come through the
// ring as they are, 128 columns 320 and 332, 144 columns 360 and 345), and its tiles give half of the pairs work (a lone expert of
// 2048 x 512: 2048 tokens 65 and 80, 4096 90 and 90; four experts of 1024 x 512 with 200 columns 37 and 41, sixteen with
// 150 48 and 44).
// One CTA, 256: above 128 columns an expert (16 experts of 1024 x 512, K = 4, ms a call, gate/up and down tiles of 128 and of 256: Q4_0 700
// tokens 1.88 and 1.37, 2000 4.20 and 3.34; Q8_0 2000 4.37 and 3.49; BF16 2000 3.15 and 2.86).
// ctas: cap of the persistent grid (0 = every SM).
struct TcForm {
    int cols;
    bool pairs;
};
inline TcForm tc_form(const LayerDev& L, int columns, int sms, int ctas) {
    if (ctas == 1) return TcForm{columns > 128 * L.E ? 256 : 128, false};
    const int least = L.gu16 != nullptr ? 136 : 120, tiles = (columns / 512 > L.E ? columns / 512 : L.E) * (L.I / 128);
    return TcForm{columns > least * L.E && 4 * tiles >= sms ? 512 : 128, true};
}

// Routing tables of one call (device pointers into the context's scratch).
struct RouteDev {
    float* logits;         // [T,E]
    uint32_t* ids;         // [T,K] selection order
    float* weights;        // [T,K]
    int32_t* expert_bounds;  // [E+1]
    int32_t* col_expert;   // [C]
    int32_t* col_src_tok;  // [C]
    int32_t* dst_to_col;   // [C] indexed t*K+slot
    int32_t* uexp;         // [E] distinct experts, ascending
    int32_t* n_uexp;       // [1]
    unsigned int* ticket;  // [1] last-block election counter (zero between launches)
    int4* work;            // [2*E] decode work descriptors: {expert | -1, first column, columns, 0}, {tok0..tok3}
};

// Activation fragments: for token (or compact column) c, half hl (0 = high part,
// 1 = low part of the f32 value split into two f16), block b, t in 0..3: one uint4
//   {pack(v[4t],v[4t+2]), pack(v[4t+1],v[4t+3]), pack(v[16+4t],v[16+4t+2]), pack(v[16+4t+1],v[16+4t+3])}
// i.e. the m16n8k16 B fragments (b0,b1) of the low-nibble MMA then of the
// high-nibble MMA of that block. Index: ((c*2 + hl)*nblk_pad + b)*4 + t.
struct DecodeArgs {
    LayerDev L;
    RouteDev R;
    const float* x;         // normed [T,H] (or raw x when gamma != null)
    const float* gamma;     // fused FFN norm weight or null
    float* normed_out;      // optional normed output when gamma != null
    float eps;
    const float* residual;  // [T,H]
    float* out;             // [T,H]
    const float* logits_override;  // [T,E] or null
    uint4* xf;              // activation fragments [T][2][kg_h*4][4]
    unsigned* xq;           // two-term int8 activations [T][xq_tok_words] of the kernel chain's Q4_0 gate/up (null = f16 fragments in xf)
    unsigned* sq;           // two-term int8 SwiGLU outputs [C][xq_tok_words(kg_i*4)]: down operand of the Q4_0 chain (null = f16 fragments in sf)
    uint4* sf;              // SwiGLU fragments     [C][2][kg_i*4][4]
    float* s_f32;           // optional [C,I] f32 copy of the SwiGLU output (null = skip)
    int T, K, gating;
    int sms;                // multiprocessors of the device
    float* d32;             // [C,H] unweighted down outputs by compact column (kernel chain)
    unsigned int* bar;      // grid barrier of the fused kernel: arrival counter + per-CTA barrier counts (1024 words); null = kernel chain
    int32_t* status;        // context status word (non-zero after a bounded wait expired)
    int32_t* status_host;   // the same code for the host: a word of mapped pinned host memory (null = none)
    unsigned wait_limit_us; // limit of every device-side wait of this launch (0 = one second)
    int debug_expire;       // test hook: the fused kernel's grid barrier expects this many arrivals more than there are CTAs, the
                            // first copy barrier of the chain this many bytes more than arrive
    unsigned long long* trace;  // optional [grid][12] globaltimer stamps of the fused kernel's phases (null = off)
};

// A decode call of the always-on shared expert: known without a router, so nothing is ranked
__host__ __device__ inline bool single_expert(const DecodeArgs& a) {
    return a.L.E == 1 && a.K == 1 && a.gating >= 2 && a.logits_override == nullptr;
}

#ifdef __CUDACC__
// A kernel that gives up records why: the first code wins; the host copy is written once.
__device__ __forceinline__ void raise_status(int32_t* status, int32_t* status_host, int code) {
    if (atomicCAS(status, 0, code) == 0 && status_host != nullptr) {
        *reinterpret_cast<volatile int32_t*>(status_host) = code;
        __threadfence_system();
    }
}

// Sum of squares of a row and its RMSNorm scale by a CTA of 256 threads, each with chunks of inputs 4t.. and 16+4t.. of
// 32-blocks: one order of summation for the norm alone and for the norm fused with what follows it.
__device__ __forceinline__ float norm_sq_chunk(float ss, const float4& p, const float4& q) {
    // (written out: left to the compiler, the contractions differ from kernel to kernel)
    auto sq4 = [](const float4& v) { return __fmaf_rn(v.w, v.w, __fmaf_rn(v.z, v.z, __fmaf_rn(v.y, v.y, __fmul_rn(v.x, v.x)))); };
    return __fadd_rn(__fadd_rn(ss, sq4(p)), sq4(q));
}
__device__ __forceinline__ float norm_scale(float ss, float* red8, int H, float eps) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red8[threadIdx.x >> 5] = ss;
    __syncthreads();
    float s = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += red8[w];
    return 1.0f / sqrtf(s / (float)H + eps);
}

// Programmatic dependent launch for the chains of small kernels around the grouped products. A
// kernel launched with launch_dep() may be scheduled while the kernel before it in the stream
// is still running; it calls grid_dep_sync() as its first statement (every thread, before any
// early return, before touching anything an earlier kernel wrote): that returns once the
// preceding kernel has completed and its writes are visible, so the order of the stream is
// kept, and because every kernel of a chain does so, completion of one implies completion of
// all before it. What overlaps is the launch itself and whatever the kernel does before the call.
__device__ __forceinline__ void grid_dep_sync() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_dep(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}
#endif

// launchers (kernels.cu files)
cudaError_t launch_repack(const uint8_t* blob, const uint64_t* d_gate_offs, const uint64_t* d_up_offs,
                          const uint64_t* d_down_offs, const LayerDev& L, uint4* q, uint4* s,
                          cudaStream_t st);
cudaError_t launch_dequant_f16(const uint8_t* blob, const uint64_t* d_gate_offs, const uint64_t* d_up_offs,
                               const uint64_t* d_down_offs, const LayerDev& L, __half* gu16, __half* dn16,
                               cudaStream_t st);
cudaError_t launch_decode(const DecodeArgs& a, cudaStream_t st);
cudaError_t launch_ep_prepare(const void* x, int act_dtype, const RouteDev& R, int C, int H, int E, int epr, void* rows,
                              int32_t* local_ids, long long* send_counts, cudaStream_t st);
cudaError_t launch_route_small(const DecodeArgs& a, cudaStream_t st);  // router + tables only (T <= 16)
bool decode_fused_applicable(const DecodeArgs& a);
bool decode_uses_fused(const DecodeArgs& a);  // whether launch_decode takes the fused kernel for this call
cudaError_t launch_decode_fused(const DecodeArgs& a, cudaStream_t st);
constexpr int FUSED_MAX_TOKENS = 4;
constexpr int FUSED_MAX_LAYERS = 64;  // layers of a stack in one launch (2 KB of kernel parameters)
cudaError_t launch_decode_fused_stack(const DecodeArgs& a, const LayerDev* const* layers, const float* const* gammas, int n,
                                      float* x_tagged, cudaStream_t st);
// one step of the kernel chain: 0 router, 1 gate/up, 2 down + combine. alone: any other step may be in front of it in the stream
cudaError_t launch_decode_phase(const DecodeArgs& a, int phase, bool alone, cudaStream_t st);
cudaError_t launch_quantize(const float* src, int64_t n, int quant, void* dst, cudaStream_t st);
cudaError_t launch_rmsnorm(const float* x, const float* gamma, float* out, int T, int H, float eps,
                           cudaStream_t st);
cudaError_t launch_debug_expf(const float* in, float* out, int64_t n, cudaStream_t st);

// prefill path
struct PrefillArgs {
    LayerDev L;
    RouteDev R;
    const void* x;          // normed [T,H], f32 or bf16
    int act_dtype;          // 0 f32, 1 bf16
    const float* gamma;     // non-null: x is the raw residual stream (f32), the activations are rmsnorm(x; gamma, eps)
    float eps;
    const float* residual;
    float* out;
    const float* logits_override;
    int T, K, gating;
    // scratch
    int32_t* blk_hist;      // [E, nchunks], then [E] totals
    __half* w16;            // [2, E, H] router weight split into f16 high and low planes (per call, when the layer has none)
    __half* xr16;           // [2, T, H] activations split into f16 high and low planes (tcgen05 router)
    float* rpart;           // [ksplit, T, E] partial logits of the tcgen05 router
    int32_t* stream_starts; // [2][sms + 1] first item of every CTA of the streaming gate/up and down kernels
    int32_t* any_lo;        // [1] some low part of the activations is non-zero
    int sms;                // multiprocessors of the device
    __half* s16;            // [C, I] f16 SwiGLU output, row-major by compact column
    __half* d16;            // [C, H] f16 down output by compact column
    int4* tiles;            // tile list for the grouped GEMMs
    int32_t* n_tiles;       // [4]: gate/up tiles, down tiles, and the two kernels' tile counters
    unsigned int* tile_counter;  // [2] dynamic tile scheduler counters
    int32_t* status;        // [1] device-side error flag (bounded waits, invalid caller-supplied ids)
    int32_t* status_host;   // the same code in mapped pinned host memory (null = none)
    unsigned wait_limit_us; // limit of the device-side waits (0 = two seconds)
    int debug_extra_tx;     // test hook: the first copy barrier of the expert products expects this many bytes more than arrive
    int tc_ctas;            // cap of the persistent tcgen05 grid (0 = every SM)
    int impl;               // 0 = tcgen05 path, 1 = mma.sync grouped fallback, 2 = streaming kernels (few columns per expert)
    const uint32_t* ids_in;  // caller-supplied routing [T,K] (null = route here)
    const float* weights_in; // [T,K] or null (= 1)
};
cudaError_t launch_route_large(const PrefillArgs& a, cudaStream_t st);
// grouped products on CTA pairs (prefill_pair.cu)
cudaError_t launch_grouped_pair(const PrefillArgs& p, const void* x16, int tile_cols, int ctas, cudaStream_t st, __half* out16_rows);
bool route_single_applicable(const PrefillArgs& a);  // one expert: launch_route_large leaves the operand plane in xr16, columns = tokens
// tcgen05 router (route_tc.cu)
cudaError_t launch_split_router_w16(const float* w, __half* w16, int E, int H, bool natural, cudaStream_t st);
// f16 planes of the activations (see route_tc.cu); any_lo null = high plane only
cudaError_t launch_split_x16(const void* x, int act_dtype, int T, int H, bool natural, __half* x16, int32_t* any_lo, cudaStream_t st);
// the planes of rmsnorm(x; gamma, eps)
bool norm_split_applicable(int H, const void* x, const void* gamma);
cudaError_t launch_norm_split(const float* x, const float* gamma, float eps, int T, int H, bool natural, __half* x16, int32_t* any_lo,
                              cudaStream_t st);
int router_tc_ksplit(int H);
bool router_tc_applicable(int T, int E, int H, const void* x);
cudaError_t launch_router_logits_tc(const __half* w16, int T, int E, int H, int ksplit, int sms, const __half* x16, int32_t* any_lo,
                                    float* part, int32_t* status, int32_t* status_host, unsigned wait_limit_us, cudaStream_t st);
constexpr int ROUTER_TC_MAX_KSPLIT = 4;

// Expert-parallel form of the grouped products: the rows of the activation operand are not this
// rank's T*K compact columns but whatever the peers pushed into its receive window, and the down
// product's output rows go back to the ranks they came from.
constexpr int MAX_EP_RANKS = 16;
struct TcPeerOut {
    const int32_t* ret_map;        // [rows] (source rank << 24) | row in that rank's return buffer; null = off
    __half* base[MAX_EP_RANKS];    // every rank's return buffer [rows_cap, H] f16 as mapped into this process
    int world;
    int rows_cap;                  // rows of a return buffer: indices are checked against it
};
struct TcPlan {
    int rows;      // rows of the activation operand = capacity the tile lists were laid out for
    int gu_cols;   // columns per gate/up tile the tile lists were built with (128 or 256)
};
// tile lists {expert, col_start, ncols, m_tile} of both grouped GEMMs from per-expert column counts
// left in R.expert_bounds[0..E) (turned into bounds in place), plus R.uexp / R.n_uexp. stream_mode (null = off): device
// word that says whether the call's work goes to the streaming kernels (chunks, starts) instead
cudaError_t launch_tile_plan(const RouteDev& R, int E, int H, int I, int rows_cap, int gu_cols, int4* tiles,
                             int32_t* n_tiles, cudaStream_t st, const int32_t* stream_mode, int4* chunks, int32_t* starts,
                             int sms);
// Most columns of a prompt that the streaming kernels take (experts: of the whole call, an expert-parallel rank's layer has
// a share of them). The line lies where the CTA-pair kernels overtake them, us replayed, streaming and pairs:
//   planes           E = 128, 2048 x 768: Q4_0 7 columns an expert 131 and 143, 8 columns 144 and 144, 10 columns 168 and 147; Q8_0 7 columns
//                    161 and 164, 8 columns 174 and 164. A lone expert of 2048 x 512: 8 columns 32.9 and 34.9, 9 columns 38.0 and 34.8
//   small planes     with up to 1536 inputs and no more items than the SMs have warps, one item's chain is the kernel's time, and it grows when
//                    some expert has a third operand of columns: 9 columns of E = 32, 1024 x 512 35.8 and 39.2 (Q4_0), 39.0 and 42.2 (Q8_0), of
//                    E = 16, 1024 x 1024 35.8 and 38.9; 11 columns of the former 43.3 and 39.0; E = 64, 1024 x 512 at 8 columns 49.3 and 51.8, at 9
//                    55.9 and 52.3; E = 64, 768 x 512 at 9 45.0 and 46.5
//   narrow planes    rows of up to 512 inputs are a short chain of copies for a streaming warp, while the pairs' set-up stays: 16 experts of
//                    512 x 256 at 8 columns 25.7 and 28.7, at 12 columns 27.7 and 28.7; 128 of them at 12 columns 42.4 and 44.2 (Q4_0), at 9
//                    columns 45.5 and 46.8, at 10 columns 49.0 and 46.7 (Q8_0); a lone one at 13 columns 24.7 and 26.6
//   f16 matrices     the pairs multiply these, four (Q4_0) or two times the bytes that the streaming kernels read from the planes, which counts
//                    where the matrices are more than 100 MB: E = 128, 2048 x 768: Q4_0 8 columns 146 and 209, 12 columns 196 and 214; Q8_0 10 columns
//                    202 and 212, 11 columns 217 and 213; E = 16, 2048 x 1408 at 11 columns 61 and 73; E = 8, 1024 x 2816 at 10 columns 48 and 52; but
//                    100 MB of E = 32, 2048 x 256 at 7 columns 47.0 and 46.0, at 8 columns 61.3 and 46.1, of E = 8, 2048 x 1024 at 9 columns 45.5 and 45.2.
//                    Many short rows again have the longer line: E = 32, 1024 x 512 at 10 columns 37.1 and 44.6, at 12 columns 45.0 and 44.7
// The same line for an expert-parallel call, whose results are one GPU's to the bit. There it costs time: its one-CTA tiles overtake
// later (2048 x 768, E = 128, one rank: Q4_0 8.1 columns 199 streaming and 222 on tiles, 10 columns 220 and 223, 11 columns 236 and 224).
// ctas: cap of the tcgen05 grid, which the streaming kernels do not have (0 = none). The line rises with the waves of gate/up tiles that the cap
// adds, up to 12 columns (Q8_0 9, a lone expert 16). 2048 x 768, E = 128, Q4_0, streaming and tiles: 9 columns on 120 CTAs 163 and 168, 12 columns on 100
// 193 and 196, on 48 194 and 359, 9 columns on one CTA 164 and 19393; a lone expert of few tiles keeps its line down to a few CTAs.
inline int stream_max_columns(const LayerDev& L, int experts, int sms, int ctas) {
    const bool q4 = L.quant == Q4_0;
    int most = 8 * experts;
    if (L.gu16 != nullptr && ((long long)experts * L.H * L.I > (1 << 24) ? experts >= 8 : experts >= 32 && L.H <= 1536)) most = (q4 ? 12 : 10) * experts;
    else if (L.H <= 512) most = experts == 1 ? 16 : (q4 ? 12 : 9) * experts;
    else if (L.H <= 1536 && experts > 1 && (long long)experts * L.I <= 256ll * sms) most = 9 * experts;  // (16 warps, items of 16 rows)
    if (ctas > 0 && ctas < sms) {
        const int tiles = 2 * experts * ((L.I + 127) / 128), ceiling = experts == 1 ? 16 : (q4 ? 12 : 9) * experts;  // (a tile of 128 rows occupies a pair)
        const int capped = most * ((tiles + ctas - 1) / ctas) / ((tiles + sms - 1) / sms);
        if (capped > most && most < ceiling) most = capped < ceiling ? capped : ceiling;
    }
    return most;
}
inline int stream_max_columns_of_any(int experts) { return 12 * experts > 16 ? 12 * experts : 16; }
// gate/up of a decode batch, expert products of short prompts (stream.cu)
cudaError_t launch_stream_gate_up(const DecodeArgs& p, cudaStream_t st);
cudaError_t launch_stream_down(const DecodeArgs& p, bool int8, bool after_gate_up, cudaStream_t st);
cudaError_t launch_stream_prefill(const PrefillArgs& p, const __half* x16, __half* out16_rows, cudaStream_t st, const TcPeerOut* peer = nullptr);
constexpr int STREAM_SHIFT = 5;
constexpr int STREAM_CHUNK = 1 << STREAM_SHIFT;  // columns of an expert that one item of the streaming kernels multiplies

void count_launch(int n = 1);

// cudaFuncSetAttribute(MaxDynamicSharedMemorySize) applies to the CURRENT device only, and one
// process may own contexts on several GPUs: the opt-in is remembered per device ordinal
// (`cache` is a function-local static of the launcher, one per kernel instantiation).
struct SmemOptIn {
    size_t bytes[64] = {};
};
template <typename Kern>
inline cudaError_t ensure_dyn_smem(Kern kern, size_t bytes, SmemOptIn& cache) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    if (bytes <= cache.bytes[device & 63]) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) cache.bytes[device & 63] = bytes;
    return e;
}

}  // namespace lumen
