"""The kernels of the prompt and batch paths at the sizes where they can go wrong: edges of column chunks and
tiles, remainders, the first and last size on each side of a dispatch rule. Against the CPU reference."""
import numpy as np
import pytest
import torch

from lumen_b200 import _lib, moe, synth
from oracle import oracle
from tests.gpu_util import TOL_REL_L2, kernels_of, make_layer, oracle_layer, pair_kernel, rel_l2

pytestmark = pytest.mark.gpu


def logits_for_counts(counts, K):
    """Logits under which expert e is the choice of counts[e] consecutive (token, slot) pairs (K distinct experts a token)."""
    E = len(counts)
    left = np.asarray(counts).copy()
    rows = []
    while left.max() > 0:
        pick = np.argsort(-left, kind="stable")[:K]
        row = np.full(E, -20.0, np.float32)
        row[pick] = np.linspace(1.0, 0.0, K)
        left[pick] -= 1
        rows.append(row)
    return torch.from_numpy(np.stack(rows)).cuda()


def check_prefill(H, I, E, K, quant, lg, act=torch.float32, kernels=False):
    """kernels: the names of the call's kernels are returned."""
    T = lg.shape[0]
    lay, meta, blob_np, sc, layer = make_layer(H, I, E, K, quant, seed=T, max_tokens=T)
    g = torch.Generator("cuda").manual_seed(T + 1)
    x = torch.randn((T, H), generator=g, device="cuda").to(act)
    res = torch.randn((T, H), generator=g, device="cuda")
    sc.set_logits_override(lg)
    out = sc.prefill(layer, x, res)
    r = sc.get_routing(T)
    o_out, o_ids, o_w = oracle_layer(blob_np, meta, lay, K, x.float().cpu().numpy(), res.cpu().numpy(), logits=lg.cpu().numpy())
    assert np.array_equal(r["ids"], o_ids)
    assert rel_l2((out - res).cpu().numpy(), o_out - res.cpu().numpy()) < TOL_REL_L2
    assert torch.equal(out, sc.prefill(layer, x, res))
    return kernels_of(lambda: sc.prefill(layer, x, res)) if kernels else None


# streaming kernels: chunks of 32 columns, operands of 8; experts with none, one, one more than an operand or a chunk
@pytest.mark.parametrize("quant", [0, 1])
@pytest.mark.parametrize("H,I", [(256, 128), (640, 384)])
def test_streaming_prefill_chunk_edges(cuda_lib, quant, H, I):
    counts = [0, 1, 7, 8, 9, 16, 17, 31, 0, 33, 2, 0, 1, 1, 1, 1]  # 128 columns: below the limit of 16 experts
    check_prefill(H, I, 16, 1, quant, logits_for_counts(counts, 1))


# the last batch on the streaming kernels and the first on the tcgen05 ones (12 | 9 columns an expert of such narrow rows), and others
@pytest.mark.parametrize("quant,T", [(1, 32), (1, 33), (0, 34), (0, 35), (0, 36), (0, 37), (1, 40), (1, 41), (1, 48), (1, 49)])
def test_prefill_on_both_sides_of_the_streaming_limit(cuda_lib, quant, T):
    check_prefill(384, 256, 16, 4, quant, synth.zipf_logits(T, 16, 3), torch.bfloat16)


# tcgen05 rings and claims: contractions of a few stages, tiles of 128 columns and on CTA pairs
@pytest.mark.parametrize("quant", [0, 1, 2])
@pytest.mark.parametrize("H,I,E,T", [(512, 512, 8, 257), (256, 1024, 8, 640), (768, 128, 4, 6200)])
def test_tcgen05_tiles_of_short_contractions(cuda_lib, quant, H, I, E, T):
    check_prefill(H, I, E, 2, quant, synth.uniform_logits(T, E, 7))


# products on CTA pairs, tiles of up to 512 columns: sets of 32..256 columns and what is left of them, one and two sets a
# tile, contractions of one, two, three and many 128-input groups (tiles claimed four, two and one ahead). Rows of 128
# inputs (down products of one group) are one tile of 128 an expert: 64 experts, so that half of the pairs have one
WIDE_COUNTS = [0, 1, 16, 31, 33, 64, 255, 256, 257, 288, 511, 512, 513, 1025, 7, 95]


@pytest.mark.parametrize("quant", [0, 1, 2])
@pytest.mark.parametrize("H,I,E", [(256, 1024, 16), (2048, 384, 16), (1536, 384, 16), (3072, 512, 16), (768, 640, 16), (256, 128, 64), (512, 128, 64)])
def test_pair_products_wide_tile_edges(cuda_lib, quant, H, I, E):
    form = check_prefill(H, I, E, 1, quant, logits_for_counts(WIDE_COUNTS * (E // 16), 1), torch.bfloat16, kernels=True)
    assert sum(pair_kernel(quant, mode, False) in k for k in form for mode in (0, 1)) == 2, form


# tiles of up to 128 columns: operands of 32..128 columns, several tiles an expert, contractions of one group and more
@pytest.mark.parametrize("quant", [0, 1, 2])
@pytest.mark.parametrize("H,I", [(256, 1024), (2048, 128), (1536, 384), (3072, 256), (768, 640)])
def test_pair_products_narrow_tile_edges(cuda_lib, quant, H, I):
    counts = [0, 1, 16, 31, 32, 33, 63, 65, 96, 97, 127, 128, 129, 257, 7, 400]
    form = check_prefill(H, I, 16, 1, quant, logits_for_counts(counts, 1), torch.bfloat16, kernels=True)
    assert sum(pair_kernel(quant, mode, True) in k for k in form for mode in (0, 1)) == 2, form


# tiles of 128 | 512: the last batch of the one and the first of the other; few experts; a grid capped at one CTA and at three
@pytest.mark.parametrize("quant,E,I,T", [(0, 16, 384, 960), (0, 16, 384, 961), (1, 16, 384, 961), (2, 16, 384, 1088), (2, 16, 384, 1089), (1, 4, 256, 600)])
def test_prefill_on_both_sides_of_the_wide_tiles(cuda_lib, quant, E, I, T):
    check_prefill(512, I, E, 2, quant, synth.zipf_logits(T, E, 5))


@pytest.mark.parametrize("quant", [0, 1, 2])
@pytest.mark.parametrize("ctas,T,E,K", [(1, 300, 16, 2), (1, 1024, 16, 2), (1, 1025, 16, 2), (1, 400, 1, 1), (3, 300, 16, 2), (3, 1100, 16, 2)])
def test_prefill_on_a_capped_grid(cuda_lib, quant, ctas, T, E, K):
    H, I = 512, 384
    lay = synth.LayerLayout(H, I, E, quant)
    blob = synth.make_layer_blob(lay, 3)
    x = torch.randn((T, H), generator=torch.Generator("cuda").manual_seed(T), device="cuda")
    outs = []
    for flags in (0, _lib.flag_tc_ctas(ctas)):
        sc = moe.allocate_moe_scratch(H, I, E, K, T, moe.SIGMOID_GATE if E == 1 else moe.SOFTMAX_RENORM, flags=flags)
        outs.append(sc.prefill(sc.prepare_layer(blob, lay.meta()), x, x))
        assert sc.poll_status() == _lib.OK
    assert torch.equal(*outs)


# f16 rows in the caller's order (top_k = 1): down products by row map on CTA pairs (tiles of 128 and of 512 columns), one CTA, the
# streaming kernels. With a weight of one and no residual the weighted sum is the same f16 row.
@pytest.mark.parametrize("quant", [0, 1, 2])
@pytest.mark.parametrize("T,ctas", [(60, 0), (700, 0), (2500, 0), (2500, 1)])
def test_routed_rows_leave_by_row_map(cuda_lib, quant, T, ctas):
    H, I, E = 512, 384, 16
    lay = synth.LayerLayout(H, I, E, quant)
    sc = moe.allocate_moe_scratch(H, I, E, 1, T, flags=_lib.flag_tc_ctas(ctas))
    layer = sc.prepare_layer(synth.make_layer_blob(lay, 3), lay.meta())
    g = torch.Generator("cuda").manual_seed(T)
    x = torch.randn((T, H), generator=g, device="cuda")
    ids = torch.randint(0, E - 3, (T,), generator=g, device="cuda", dtype=torch.int32)  # two experts get no row
    ids[:1], ids[1:32] = E - 3, 2
    rows16 = sc.experts_routed_f16(layer, x, ids)
    want = sc.prefill_routed(layer, x, ids, None, torch.zeros_like(x))
    assert sc.poll_status() == _lib.OK
    assert want.abs().sum(1).min() > 0 and torch.equal(rows16.float(), want)


# batches of the decode chain for each format, at contractions with a remainder against the ring's chunk
@pytest.mark.parametrize("quant,T", [(0, 3), (0, 16), (1, 5), (1, 16), (2, 5), (2, 9), (2, 16)])
def test_decode_chain_wide_layer(cuda_lib, quant, T):
    H, I, E, K = 4096, 1408, 8, 2
    lay, meta, blob_np, sc, layer = make_layer(H, I, E, K, quant, seed=T)
    g = torch.Generator("cuda").manual_seed(T)
    x = torch.randn((T, H), generator=g, device="cuda")
    gamma = 1 + 0.1 * torch.randn(H, generator=g, device="cuda")
    normed = torch.empty_like(x)
    out = sc.decode_fused_norm(layer, x, gamma, 1e-6, normed)
    r = sc.get_routing(T)
    o_normed = oracle.rmsnorm(x.cpu().numpy(), gamma.cpu().numpy(), 1e-6)
    np.testing.assert_allclose(normed.cpu().numpy(), o_normed, rtol=2e-6, atol=1e-7)
    o_out, _, _ = oracle.moe_layer(blob_np, 0, meta.expert_gate_offs, meta.expert_up_offs, meta.expert_down_offs, quant, H, I,
                                   E, K, o_normed, x.cpu().numpy(), ids=r["ids"], weights=r["weights"], threads=8)
    assert rel_l2((out - x).cpu().numpy(), o_out - x.cpu().numpy()) < TOL_REL_L2


# BF16 batches of few experts (warps by the rounds of items: test_gpu_kernel_choice.py)
@pytest.mark.parametrize("H,I,T", [(2048, 512, 6), (2048, 512, 7), (512, 2048, 3), (512, 2048, 4)])
def test_decode_chain_bf16_warp_rules(cuda_lib, H, I, T):
    E, K = 16, 8 if H < I else 4
    lay, meta, blob_np, sc, layer = make_layer(H, I, E, K, 2, seed=T)
    g = torch.Generator("cuda").manual_seed(T)
    x = torch.randn((T, H), generator=g, device="cuda")
    res = torch.randn((T, H), generator=g, device="cuda")
    out = sc.decode(layer, x, res)
    r = sc.get_routing(T)
    o_out, _, _ = oracle.moe_layer(blob_np, 0, meta.expert_gate_offs, meta.expert_up_offs, meta.expert_down_offs, 2, H, I, E, K,
                                   x.cpu().numpy(), res.cpu().numpy(), ids=r["ids"], weights=r["weights"], threads=8)
    assert rel_l2((out - res).cpu().numpy(), o_out - res.cpu().numpy()) < TOL_REL_L2


# the small router with one and with two rows of experts a warp, at widths with a remainder
@pytest.mark.parametrize("E,H,T", [(256, 1024, 5), (256, 2080, 16), (128, 4096, 7), (8, 320, 16)])
def test_small_router_rows(cuda_lib, E, H, T):
    K = min(8, E)
    lay, meta, blob_np, sc, layer = make_layer(H, 128, E, K, 1, seed=E, max_tokens=T)
    x = torch.randn((T, H), generator=torch.Generator("cuda").manual_seed(T), device="cuda")
    ids, w, lg = sc.route_only(layer, x, want_logits=True)
    router = blob_np[:lay.router_bytes].view(np.float32).reshape(E, H)
    np.testing.assert_allclose(lg.cpu().numpy(), x.cpu().numpy().astype(np.float64) @ router.T.astype(np.float64), rtol=0, atol=5e-5)
    o_ids, o_w = oracle.topk_from_logits(lg.cpu().numpy(), K, 0)
    assert np.array_equal(ids.cpu().numpy().astype(np.uint32), o_ids)
    assert np.array_equal(w.cpu().numpy().view(np.uint32), o_w.view(np.uint32))


# one CTA sorts up to 2048 pairs, the general chain more; experts beyond one warp's 128
@pytest.mark.parametrize("T,E,K", [(256, 128, 8), (257, 128, 8), (2048, 16, 1), (2049, 16, 1), (129, 256, 16), (700, 33, 5), (512, 256, 8), (2050, 255, 2)])
def test_sorting_on_both_sides_of_one_cta(cuda_lib, T, E, K):
    lg = synth.zipf_logits(T, E, T)
    sc = moe.allocate_moe_scratch(256, 128, E, K, T)
    ids, w = sc.topk_from_logits(lg)
    r = sc.get_routing(T)
    o_ids, o_w = oracle.topk_from_logits(lg.cpu().numpy(), K, 0)
    assert np.array_equal(ids.cpu().numpy().astype(np.uint32), o_ids)
    assert np.array_equal(w.cpu().numpy().view(np.uint32), o_w.view(np.uint32))
    ce, cst, d2c, bounds = oracle.counting_sort(o_ids, E)
    assert np.array_equal(r["dst_to_col"], d2c) and np.array_equal(r["col_src_tok"], cst) and np.array_equal(r["expert_bounds"], bounds)


# tcgen05 router: a token's logits are the same in tiles of 32 and of 128 tokens
@pytest.mark.parametrize("E", [128, 256])
def test_router_tiles_of_32_and_128_tokens_agree(cuda_lib, E):
    H, T = 512, 6100
    lay = synth.LayerLayout(H, 128, E, 1)
    sc = moe.allocate_moe_scratch(H, 128, E, 8, T)
    layer = sc.prepare_router_only(synth.make_layer_blob(lay, 9), lay.meta().router_weight_off)
    x = torch.randn((T, H), generator=torch.Generator("cuda").manual_seed(1), device="cuda")
    _, _, big = sc.route_only(layer, x, want_logits=True)
    for lo, hi in ((0, 31), (33, 98), (6000, 6100)):
        _, _, lg = sc.route_only(layer, x[lo:hi].contiguous(), want_logits=True)
        assert torch.equal(lg, big[lo:hi])


# every width of a router tile (64, 128 and 256 tokens beside the 32 of a few rows)
@pytest.mark.parametrize("E", [128, 256])
def test_router_tiles_of_every_width_agree(cuda_lib, E):
    H, T = 256, 4600
    lay = synth.LayerLayout(H, 128, E, 1)
    sc = moe.allocate_moe_scratch(H, 128, E, 8, T)
    layer = sc.prepare_router_only(synth.make_layer_blob(lay, 9), lay.meta().router_weight_off)
    x = torch.randn((T, H), generator=torch.Generator("cuda").manual_seed(1), device="cuda")
    parts = [sc.route_only(layer, x[t:t + 23].contiguous(), want_logits=True)[2].clone() for t in range(0, T, 23)]
    ref = torch.cat(parts)
    for n in (700, 1000, 1400, 1700, 2300, T):
        assert torch.equal(sc.route_only(layer, x[:n].contiguous(), want_logits=True)[2], ref[:n])


# two rows a CTA: an odd number of them
@pytest.mark.parametrize("H", [256, 2048])
def test_norm_folded_into_the_planes_of_a_large_batch(cuda_lib, H):
    T, E, K = 4097, 16, 2
    lay = synth.LayerLayout(H, 128, E, 1)
    sc = moe.allocate_moe_scratch(H, 128, E, K, T)
    layer = sc.prepare_layer(synth.make_layer_blob(lay, 1), lay.meta())
    g = torch.Generator("cuda").manual_seed(H)
    gamma = 1 + 0.1 * torch.randn(H, generator=g, device="cuda")
    x = torch.randn((T, H), generator=g, device="cuda")
    y = sc.prefill(layer, moe.rmsnorm(x, gamma, 1e-6), x)
    sc.stack_prefill([layer, layer], [gamma, gamma], x, 1e-6)
    assert torch.equal(x, sc.prefill(layer, moe.rmsnorm(y, gamma, 1e-6), y))


# the norm that is folded into the operand planes: one to four register chunks a row, whole and partial
@pytest.mark.parametrize("H", [512, 2048, 2304, 4096, 6400, 8192])
def test_norm_folded_into_the_planes_matches_the_norm_kernel(cuda_lib, H):
    T, E, K = 33, 16, 2
    lay = synth.LayerLayout(H, 128, E, 1)
    sc = moe.allocate_moe_scratch(H, 128, E, K, T)
    layers = [sc.prepare_layer(synth.make_layer_blob(lay, s), lay.meta()) for s in (1, 2)]
    g = torch.Generator("cuda").manual_seed(H)
    gammas = [1 + 0.1 * torch.randn(H, generator=g, device="cuda") for _ in layers]
    x0 = torch.randn((T, H), generator=g, device="cuda")
    x = x0.clone()
    sc.stack_prefill(layers, gammas, x, 1e-6)
    y = x0
    for layer, gamma in zip(layers, gammas):
        y = sc.prefill(layer, moe.rmsnorm(y, gamma, 1e-6), y)
    assert torch.equal(x, y)


# a context of one expert: routing, operand plane and plan in one kernel of 8 tokens a CTA, then streaming up to 8 columns (BF16
# none), CTA pairs beyond (9728: tiles of 512 columns)
@pytest.mark.parametrize("quant", [0, 1, 2])
@pytest.mark.parametrize("T,act,gating", [(1, torch.float32, 2), (8, torch.float32, 2), (9, torch.bfloat16, 2), (16, torch.float32, 3), (17, torch.bfloat16, 2),
                                          (129, torch.float32, 3), (9500, torch.bfloat16, 2), (9728, torch.float32, 2)])
def test_single_expert_prefill(cuda_lib, quant, T, act, gating):
    H, I = 768, 256
    lay, meta, blob_np, sc, layer = make_layer(H, I, 1, 1, quant, seed=T, max_tokens=T, gating=gating)
    g = torch.Generator("cuda").manual_seed(T)
    x = torch.randn((T, H), generator=g, device="cuda").to(act)
    res = torch.randn((T, H), generator=g, device="cuda")
    out = sc.prefill(layer, x, res)
    o_out, _, _ = oracle.moe_layer(blob_np, int(meta.router_weight_off), meta.expert_gate_offs, meta.expert_up_offs, meta.expert_down_offs,
                                   quant, H, I, 1, 1, x.float().cpu().numpy(), res.cpu().numpy(), gating=gating,
                                   threads=oracle.hardware_threads())
    assert rel_l2((out - res).cpu().numpy(), o_out - res.cpu().numpy()) < TOL_REL_L2
    r = sc.get_routing(T)
    assert (r["ids"] == 0).all() and np.array_equal(r["dst_to_col"].ravel(), np.arange(T))
    if T > 16:
        names = kernels_of(lambda: sc.prefill(layer, x, res))
        assert sum(pair_kernel(quant, mode, T < 9728) in k for k in names for mode in (0, 1)) == 2, names


# the fused decode kernel on one expert: no router exchange; items on some CTAs, on all, more than one each, ragged groups
@pytest.mark.parametrize("quant", [0, 1, 2])
@pytest.mark.parametrize("H,I,T,gating", [(2048, 512, 3, 2), (96, 160, 1, 2), (1024, 2816, 4, 3), (256, 4800, 2, 2)])
def test_single_expert_fused_decode(cuda_lib, quant, H, I, T, gating):
    lay, meta, blob_np, sc, layer = make_layer(H, I, 1, 1, quant, seed=T, gating=gating)
    g = torch.Generator("cuda").manual_seed(T)
    x = torch.randn((T, H), generator=g, device="cuda")
    res = torch.randn((T, H), generator=g, device="cuda")
    o_out, _, o_w = oracle.moe_layer(blob_np, int(meta.router_weight_off), meta.expert_gate_offs, meta.expert_up_offs, meta.expert_down_offs,
                                     quant, H, I, 1, 1, x.cpu().numpy(), res.cpu().numpy(), gating=gating, threads=oracle.hardware_threads())
    outs = [sc.decode(layer, x, res).clone() for _ in range(10)]
    assert rel_l2((outs[0] - res).cpu().numpy(), o_out - res.cpu().numpy()) < TOL_REL_L2
    assert all(torch.equal(o, outs[0]) for o in outs)
    r = sc.get_routing(T)
    assert (r["ids"] == 0).all() and np.array_equal(r["dst_to_col"].ravel(), np.arange(T)) and np.array_equal(r["expert_bounds"], [0, T])
    np.testing.assert_allclose(r["weights"], o_w, rtol=1e-4)


# a one-token stack of Q4_0 layers in one launch: more layers than one launch holds, other formats in between, CTAs with
# and without down rows, more experts than CTAs; other formats, more tokens, a captured stream: layer by layer
@pytest.mark.parametrize("quants,H,E,T", [([1] * 66, 256, 16, 1), ([0, 0, 1, 1, 2, 2, 2, 0], 512, 16, 1), ([1] * 5, 2048, 256, 1),
                                          ([1] * 4, 1920, 128, 1), ([0, 2, 1, 1], 128, 8, 1), ([1] * 5, 2048, 16, 3), ([0] * 4, 1920, 256, 2), ([1] * 3, 256, 16, 5)])
def test_fused_stack_matches_layer_by_layer(cuda_lib, quants, H, E, T):
    I, K = 128, 4
    sc = moe.allocate_moe_scratch(H, I, E, K, 16)
    layers = []
    for l, quant in enumerate(quants):
        lay = synth.LayerLayout(H, I, E, quant)
        layers.append(sc.prepare_layer(synth.make_layer_blob(lay, l), lay.meta()))
    g = torch.Generator("cuda").manual_seed(H)
    gammas = [1 + 0.1 * torch.randn(H, generator=g, device="cuda") for _ in layers]
    x0 = torch.randn((T, H), generator=g, device="cuda")
    y = x0.clone()
    for layer, gamma in zip(layers, gammas):
        y = sc.decode_fused_norm(layer, y, gamma, 1e-6, torch.empty_like(y))
    for _ in range(20):
        x = x0.clone()
        sc.stack_decode(layers, gammas, x, 1e-6)
        assert torch.equal(x, y)
    assert sc.poll_status() == 0
    graph = torch.cuda.CUDAGraph()  # captured: one launch per layer
    x.copy_(x0)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        sc.stack_decode(layers, gammas, x, 1e-6)
    assert torch.equal(x, x0)
    graph.replay()
    assert torch.equal(x, y)


# weighted sum of the expert outputs: rows of no whole number of 16-byte words, buffers between two 16-byte boundaries
@pytest.mark.parametrize("H", [2, 6, 8, 36, 514, 2048])
@pytest.mark.parametrize("off", [0, 1])
def test_combine_of_any_even_width_and_4_byte_boundary(cuda_lib, H, off):
    T, K = 5, 3
    g = torch.Generator("cuda").manual_seed(H)
    d16 = torch.randn((T * K, H), generator=g, device="cuda").half()
    w = torch.rand((T, K), generator=g, device="cuda")
    d2c = torch.randperm(T * K, generator=g, device="cuda").int()
    pad = torch.full((2, T * H + 8), 7.0, device="cuda")  # words around the rows that no thread may touch
    res, out = (p[off:off + T * H].view(T, H) for p in pad)
    res.copy_(torch.randn((T, H), generator=g, device="cuda"))
    want = res.clone()
    for s in range(K):  # slot order, product and sum rounded apart
        want = want + w[:, s:s + 1] * d16[d2c.view(T, K)[:, s].long()].float()
    moe.combine_f16(d16, res, w, d2c, out)
    assert torch.equal(out, want)
    assert (pad[:, :off] == 7.0).all() and (pad[:, off + T * H:] == 7.0).all()


# prompts whose residual and output lie on a 4-byte boundary: streaming, tcgen05 and mma.sync products
@pytest.mark.parametrize("H,I,T", [(512, 256, 20), (512, 256, 200), (160, 96, 50)])
def test_prefill_residual_and_output_on_a_4_byte_boundary(cuda_lib, H, I, T):
    E, K = 16, 4
    _, _, _, sc, layer = make_layer(H, I, E, K, 1, seed=T, max_tokens=T)
    g = torch.Generator("cuda").manual_seed(T)
    x = torch.randn((T, H), generator=g, device="cuda")
    res = torch.randn((T, H), generator=g, device="cuda")
    aligned = sc.prefill(layer, x, res)
    pad = torch.full((2, T * H + 2), 7.0, device="cuda")
    res_odd, out_odd = (p[1:-1].view(T, H) for p in pad)
    res_odd.copy_(res)
    assert torch.equal(sc.prefill(layer, x, res_odd, out_odd), aligned)
    sc.prefill(layer, x, res_odd, res_odd)
    assert torch.equal(res_odd, aligned) and (pad[:, 0] == 7.0).all() and (pad[:, -1] == 7.0).all()
