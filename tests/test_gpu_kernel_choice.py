"""Which kernels a call takes: both sides of the lines that the host draws by shapes, formats and columns per expert."""
import pytest
import torch

from lumen_b200 import _lib, moe, synth
from tests.gpu_util import TOL_REL_L2, kernels_of, rel_l2

pytestmark = pytest.mark.gpu


def context(H, I, E, K, quant, T, flags=0):
    lay = synth.LayerLayout(H, I, E, quant)
    sc = moe.allocate_moe_scratch(H, I, E, K, max(T, 16), moe.SIGMOID_GATE if E == 1 else moe.SOFTMAX_RENORM, flags=flags)
    return sc, sc.prepare_layer(synth.make_layer_blob(lay, 5), lay.meta())


def rows(T, H):
    return torch.randn((T, H), generator=torch.Generator("cuda").manual_seed(T), device="cuda")


# streaming down product of Q4_0 prompts: 24 warps for enough items (E * H / 16 rows of tiles) and more than two columns of long rows, 4.5
# to 6 columns of short ones; 16 elsewhere
@pytest.mark.parametrize("H,I,E,K,T,warps", [(1024, 1024, 256, 2, 256, 16), (1024, 1024, 256, 2, 257, 24), (1024, 1024, 256, 2, 1024, 24),
                                             (1024, 1024, 128, 2, 300, 16), (1024, 128, 256, 2, 576, 16), (1024, 128, 256, 2, 577, 24),
                                             (1024, 128, 256, 2, 768, 24), (1024, 128, 256, 2, 769, 16), (1024, 2048, 1, 1, 8, 16)])
def test_warps_of_a_prompts_streaming_down_product(cuda_lib, H, I, E, K, T, warps):
    sc, layer = context(H, I, E, K, 1, T)
    x = rows(T, H)
    out = torch.empty_like(x)
    names = kernels_of(lambda: sc.prefill(layer, x, x, out))
    assert [k for k in names if f"stream_kernel<1, 1, {warps}>" in k] and sum("stream_kernel<1, 1," in k for k in names) == 1, names
    ref, ref_layer = context(H, I, E, K, 1, T, _lib.FLAG_PREFILL_MMA)
    want = ref.prefill(ref_layer, x, x)
    assert rel_l2((out - x).cpu(), (want - x).cpu()) < TOL_REL_L2


# an expert-parallel call: by its own columns, not by what its window could take
@pytest.mark.parametrize("T,warps", [(2, 16), (256, 16), (257, 24)])
def test_warps_of_an_expert_parallel_streaming_down_product(cuda_lib, T, warps):
    from lumen_b200 import ep
    H, I, E, K = 1024, 1024, 256, 2
    lay = synth.LayerLayout(H, I, E, 1)
    pe = ep.PushExpertParallel(H, I, E, K, 1024, 0, 1, 0)
    layer = pe.prepare_layer(synth.make_layer_blob(lay, 5), lay.meta())
    x = rows(T, H)
    names = kernels_of(lambda: pe.forward(layer, x, x))
    assert [k for k in names if f"stream_kernel<1, 1, {warps}>" in k] and sum("stream_kernel<1, 1," in k for k in names) == 1, names
    pe.close()
