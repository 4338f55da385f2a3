"""Which kernels a call takes: both sides of the lines that the host draws by shapes, formats and columns per expert."""
import pytest
import torch

from lumen_b200 import _lib, moe, synth
from tests.gpu_util import TOL_REL_L2, kernels_of, rel_l2

pytestmark = pytest.mark.gpu

F16 = _lib.FLAG_PREFILL_F16_WEIGHTS


def context(H, I, E, K, quant, T, flags=0):
    lay = synth.LayerLayout(H, I, E, quant)
    sc = moe.allocate_moe_scratch(H, I, E, K, max(T, 16), moe.SIGMOID_GATE if E == 1 else moe.SOFTMAX_RENORM, flags=flags)
    return sc, sc.prepare_layer(synth.make_layer_blob(lay, 5), lay.meta())


def rows(T, H):
    return torch.randn((T, H), generator=torch.Generator("cuda").manual_seed(T), device="cuda")


# streaming down product of Q4_0 prompts: 16 warps whatever the columns, whose distribution over the experts the host does not know
@pytest.mark.parametrize("I,E,K,T,flags", [(1024, 256, 2, 256, 0), (1024, 256, 2, 257, 0), (1024, 256, 2, 1024, 0), (1024, 256, 2, 1152, F16),
                                           (128, 256, 2, 577, 0), (128, 256, 2, 768, 0), (2048, 1, 1, 8, 0)])
def test_warps_of_a_prompts_streaming_down_product(cuda_lib, I, E, K, T, flags):
    H = 1024
    sc, layer = context(H, I, E, K, 1, T, flags)
    x = rows(T, H)
    out = torch.empty_like(x)
    names = kernels_of(lambda: sc.prefill(layer, x, x, out))
    assert [k for k in names if "stream_kernel<1, 1, 16>" in k] and sum("stream_kernel<1, 1," in k for k in names) == 1, names
    ref, ref_layer = context(H, I, E, K, 1, T, _lib.FLAG_PREFILL_MMA)
    want = ref.prefill(ref_layer, x, x)
    assert rel_l2((out - x).cpu(), (want - x).cpu()) < TOL_REL_L2


# the longest prompt on the streaming kernels: planes (8 columns an expert), small ones (9), narrow ones (12 | 9, a lone expert 16), layers
# kept as f16 matrices (12 | 10 where these are many bytes or many short rows, else as planes)
@pytest.mark.parametrize("quant,flags,H,E,K,T", [(1, 0, 2048, 16, 4, 32), (0, 0, 2048, 16, 4, 32), (1, 0, 1024, 16, 4, 36), (0, 0, 1024, 16, 4, 36),
                                                 (1, 0, 1024, 256, 4, 512), (1, 0, 512, 16, 4, 48), (0, 0, 512, 16, 4, 36),
                                                 (1, F16, 1024, 32, 4, 96), (0, F16, 1024, 32, 4, 80), (1, F16, 1024, 16, 4, 36), (1, F16, 2048, 64, 4, 192),
                                                 (0, F16, 2048, 64, 4, 160), (1, F16, 2048, 32, 4, 64), (1, 0, 1024, 1, 1, 8), (0, 0, 512, 1, 1, 16)])
def test_longest_prompt_on_the_streaming_kernels(cuda_lib, quant, flags, H, E, K, T):
    I = 256
    sc, layer = context(H, I, E, K, quant, T + 1, flags)
    ref, ref_layer = context(H, I, E, K, quant, T + 1, _lib.FLAG_PREFILL_MMA)
    for n, name in ((T, "stream_kernel"), (T + 1, "grouped_gemm_pair_kernel")):
        x = rows(n, H)
        out = torch.empty_like(x)
        names = kernels_of(lambda: sc.prefill(layer, x, x, out))
        assert [k for k in names if "stream_kernel" in k or "grouped_gemm" in k or "down" in k] and all(
            name in k for k in names if "stream_kernel" in k or "grouped_gemm" in k), names
        want = ref.prefill(ref_layer, x, x)
        assert rel_l2((out - x).cpu(), (want - x).cpu()) < TOL_REL_L2


# ... where the tcgen05 grid is capped: 12 | 9 columns and a lone expert 16 on a few CTAs, 9 columns on nearly all
@pytest.mark.parametrize("ctas,quant,flags,E,K,T,tiles", [(1, 1, 0, 16, 4, 48, "tc"), (1, 0, 0, 16, 4, 36, "tc"), (1, 1, F16, 16, 4, 48, "tc"), (1, 1, 0, 1, 1, 16, "tc"),
                                                          (2, 1, 0, 16, 4, 48, "pair"), (24, 1, 0, 16, 4, 48, "pair"), (146, 1, 0, 16, 4, 36, "pair"),
                                                          (48, 1, 0, 1, 1, 8, "pair")])
def test_longest_prompt_on_the_streaming_kernels_beside_a_capped_grid(cuda_lib, ctas, quant, flags, E, K, T, tiles):
    H, I = 1024, 256
    sc, layer = context(H, I, E, K, quant, T + 1, flags | _lib.flag_tc_ctas(ctas))
    ref, ref_layer = context(H, I, E, K, quant, T + 1, _lib.FLAG_PREFILL_MMA)
    for n, name in ((T, "stream_kernel"), (T + 1, f"grouped_gemm_{tiles}_kernel")):
        x = rows(n, H)
        out = torch.empty_like(x)
        names = kernels_of(lambda: sc.prefill(layer, x, x, out))
        assert sum(name in k for k in names if "stream_kernel" in k or "grouped_gemm" in k) == 2, names
        want = ref.prefill(ref_layer, x, x)
        assert rel_l2((out - x).cpu(), (want - x).cpu()) < TOL_REL_L2


# an expert-parallel call on a capped grid draws the one-GPU line of its planes: the same bits on both sides of it
@pytest.mark.parametrize("T", [40, 48, 49])
def test_expert_parallel_call_beside_a_capped_grid(cuda_lib, T):
    from lumen_b200 import ep
    H, I, E, K, flags = 1024, 256, 16, 4, _lib.flag_tc_ctas(1)
    sc, layer = context(H, I, E, K, 1, T, flags)
    lay = synth.LayerLayout(H, I, E, 1)
    pe = ep.PushExpertParallel(H, I, E, K, 64, 0, 1, 0, flags=flags)
    pe_layer = pe.prepare_layer(synth.make_layer_blob(lay, 5), lay.meta())
    x = rows(T, H)
    want, got = sc.prefill(layer, x, x), pe.forward(pe_layer, x, x)
    assert pe.sc.poll_status() == _lib.OK and torch.equal(got, want)
    pe.close()


# decode batches: more warps where an SM's items take a round less with them (gate/up of BF16 8 | 10, down of Q8_0 16 | 20, of BF16 8 | 12), of
# Q4_0 (down on int8, its gate/up kernel has one form) from ten items on
@pytest.mark.parametrize("quant,H,I,E,K,T,gate_up,down", [(2, 2048, 768, 128, 8, 4, 10, 12), (2, 2048, 768, 128, 8, 5, 8, 12), (2, 2048, 512, 256, 8, 5, 10, 12),
                                                          (2, 2048, 512, 256, 8, 16, 8, 12), (2, 2048, 768, 128, 8, 16, 8, 8), (2, 4096, 1536, 64, 6, 9, 8, 8), (2, 1024, 384, 64, 4, 12, 8, 8),
                                                          (0, 2048, 768, 128, 8, 3, 16, 20), (0, 2048, 768, 128, 8, 4, 16, 16),
                                                          (0, 2048, 768, 128, 8, 6, 16, 20), (0, 2048, 768, 128, 8, 16, 16, 16),
                                                          (0, 2048, 1408, 64, 6, 12, 16, 20), (0, 2048, 1408, 64, 6, 13, 16, 16), (0, 4096, 1536, 64, 6, 2, 16, 16),
                                                          (1, 1024, 2816, 1, 1, 11, 0, 16), (1, 1024, 2816, 8, 2, 15, 0, 16), (1, 1024, 512, 32, 4, 9, 0, 16),
                                                          (1, 1024, 512, 32, 4, 14, 0, 20), (1, 2048, 768, 128, 8, 16, 0, 20)])
def test_warps_of_a_decode_batch(cuda_lib, quant, H, I, E, K, T, gate_up, down):
    sc, layer = context(H, I, E, K, quant, T, _lib.FLAG_DECODE_SPLIT)
    x = rows(T, H)
    out = torch.empty_like(x)
    names = kernels_of(lambda: sc.decode(layer, x, x, out))
    for mode, warps in ((4, down),) if quant == 1 else ((2, gate_up), (3, down)):
        assert [k for k in names if f"stream_kernel<{quant}, {mode}, {warps}>" in k], names
    ref, ref_layer = context(H, I, E, K, quant, T, _lib.FLAG_PREFILL_MMA)
    want = ref.prefill(ref_layer, x, x)
    assert rel_l2((out - x).cpu(), (want - x).cpu()) < TOL_REL_L2


# tcgen05 products on a grid capped at one CTA: tiles of 256 columns above 128 columns an expert
@pytest.mark.parametrize("quant,flags,T,cols", [(2, 0, 1025, 256), (2, 0, 1024, 128), (1, F16, 1025, 256), (1, 0, 1025, 256), (0, 0, 1024, 128)])
def test_gate_up_tiles_of_one_cta(cuda_lib, quant, flags, T, cols):
    sc, layer = context(512, 384, 16, 2, quant, T, flags | _lib.flag_tc_ctas(1))
    x = rows(T, 512)
    names = kernels_of(lambda: sc.prefill(layer, x, x))
    for mode in (0, 1):
        assert [k for k in names if "grouped_gemm_tc_kernel" in k and f", {mode}, {cols}," in k], names


# tokens per tile of the tcgen05 router: by bytes and waves of CTAs, 128 instead of 64 where these fill most SMs, instead of 256 where its second wave is short
@pytest.mark.parametrize("E,T,width", [(128, 100, 32), (128, 1000, 32), (128, 1500, 64), (128, 1800, 128), (128, 4096, 128), (128, 6000, 256),
                                       (256, 832, 64), (256, 1000, 128), (256, 2500, 128), (256, 3000, 256)])
def test_router_tile_width(cuda_lib, E, T, width):
    lay = synth.LayerLayout(2048, 128, E, 1)
    sc = moe.allocate_moe_scratch(2048, 128, E, 8, T)
    layer = sc.prepare_router_only(synth.make_layer_blob(lay, 9), lay.meta().router_weight_off)
    x = rows(T, 2048)
    names = kernels_of(lambda: sc.route_only(layer, x))
    assert [k for k in names if f"router_logits_tc_kernel<{width}>" in k], names


# rows gathered by column are kept only where a kernel reads them: a grid capped at one CTA
def test_device_memory_of_a_prefill_context(cuda_lib):
    H, K, T = 2048, 8, 8192
    taken = {}
    for ctas in (1, 0, 2):
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        sc = moe.allocate_moe_scratch(H, 128, 16, K, T, flags=_lib.flag_tc_ctas(ctas))
        taken[ctas] = free - torch.cuda.mem_get_info()[0]
        sc.close()
    # (the driver maps device memory in pages of 2 MB)
    assert abs(taken[1] - taken[0] - T * K * H * 2) <= 4 << 20 and abs(taken[0] - taken[2]) <= 4 << 20, taken
