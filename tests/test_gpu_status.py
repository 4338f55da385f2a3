"""Error path of the operator, through the C ABI: a kernel that gives up must be visible to
the host without a debug readback (the reference returns Result<(), RuntimeError> from every
launch, error.rs:6-31, cuda/moe.rs:1497-1502), and the context must be usable again after a
reset. The waits are made to run out from the host side: the kernel is told to expect one
arrival (or one byte) more than can come, with the limit shortened to 2 ms. Nothing here
faults, traps or hangs the GPU."""
import numpy as np
import pytest
import torch

from lumen_b200 import _lib, moe, synth
from oracle import oracle
from tests.gpu_util import kernels_of, pair_kernel

pytestmark = pytest.mark.gpu


def _ctx(H, I, E, K, max_tokens, flags=0, device=0):
    lay = synth.LayerLayout(H, I, E, 1)
    blob = synth.make_layer_blob(lay, 0, device=f"cuda:{device}")
    sc = moe.allocate_moe_scratch(H, I, E, K, max_tokens, device=device, flags=flags)
    return lay, blob, sc, sc.prepare_layer(blob, lay.meta())


def test_decode_grid_barrier_that_runs_out_is_reported_and_recoverable(cuda_lib):
    H, I, E, K, T = 512, 256, 32, 4, 2
    _, blob, sc, layer = _ctx(H, I, E, K, 16, flags=_lib.FLAG_SHORT_WAITS)
    x = torch.randn((T, H), generator=torch.Generator("cuda").manual_seed(3), device="cuda")
    good = sc.decode(layer, x, x.clone()).clone()
    torch.cuda.synchronize()
    assert sc.poll_status() == _lib.OK
    sc.debug_expire_next_wait(0)
    sc.decode(layer, x, x.clone())           # every CTA's wait at the second grid barrier runs out
    torch.cuda.synchronize()
    assert sc.poll_status() == _lib.TIMEOUT  # no readback needed: the kernel told the host
    with pytest.raises(moe.LumenMoeError) as ei:
        sc.decode(layer, x, x.clone())       # entry points fail instead of launching on a failed context
    assert ei.value.code == _lib.TIMEOUT
    with pytest.raises(moe.LumenMoeError) as ei:
        sc.get_routing(T)                    # reports it once and resets the context
    assert ei.value.code == _lib.TIMEOUT
    assert sc.poll_status() == _lib.OK
    again = sc.decode(layer, x, x.clone())
    # bit-identical to a context that never failed
    _, _, sc2, layer2 = _ctx(H, I, E, K, 16)
    fresh = sc2.decode(layer2, x, x.clone())
    torch.cuda.synchronize()
    assert torch.equal(again, good) and torch.equal(again, fresh)


def test_grouped_gemm_stage_barrier_that_runs_out_is_reported_and_recoverable(cuda_lib):
    H, I, E, K, T = 512, 256, 16, 4, 200
    _, blob, sc, layer = _ctx(H, I, E, K, T, flags=_lib.FLAG_SHORT_WAITS)
    g = torch.Generator("cuda").manual_seed(4)
    x = torch.randn((T, H), generator=g, device="cuda").to(torch.bfloat16)
    res = torch.randn((T, H), generator=g, device="cuda")
    good = sc.prefill(layer, x, res).clone()
    torch.cuda.synchronize()
    sc.debug_expire_next_wait(1)
    sc.prefill(layer, x, res)                # the first stage of the gate/up GEMM never completes
    torch.cuda.synchronize()
    assert sc.poll_status() == _lib.TIMEOUT
    with pytest.raises(moe.LumenMoeError) as ei:
        sc.prefill(layer, x, res)
    assert ei.value.code == _lib.TIMEOUT
    sc.clear_status()
    assert sc.poll_status() == _lib.OK
    again = sc.prefill(layer, x, res)
    torch.cuda.synchronize()
    assert torch.equal(again, good)


# the same on CTA pairs (both CTAs give up), tiles of 128 columns (I = 256: too few of 512) and of 512, dequantised and TMA-fed weights
@pytest.mark.parametrize("quant", [0, 1, 2])
@pytest.mark.parametrize("I,narrow", [(256, True), (640, False)])
def test_pair_stage_barrier_that_runs_out_is_reported_and_recoverable(cuda_lib, quant, I, narrow):
    H, E, K, T = 2048, 8, 2, 1500
    lay = synth.LayerLayout(H, I, E, quant)
    sc = moe.allocate_moe_scratch(H, I, E, K, T, flags=_lib.FLAG_SHORT_WAITS)
    layer = sc.prepare_layer(synth.make_layer_blob(lay, 0), lay.meta())
    x = torch.randn((T, H), generator=torch.Generator("cuda").manual_seed(4), device="cuda")
    good = sc.prefill(layer, x, x).clone()
    names = kernels_of(lambda: sc.prefill(layer, x, x))
    assert sum(pair_kernel(quant, mode, narrow) in k for k in names for mode in (0, 1)) == 2, names
    assert sc.poll_status() == _lib.OK
    sc.debug_expire_next_wait(1)
    sc.prefill(layer, x, x)
    torch.cuda.synchronize()
    assert sc.poll_status() == _lib.TIMEOUT
    sc.clear_status()
    assert torch.equal(sc.prefill(layer, x, x), good)


# the streaming kernels: decode chains on int8 (Q4_0) and hi + lo operands, short prompts
@pytest.mark.parametrize("call,quant,T", [("decode", 1, 16), ("decode", 0, 5), ("decode", 2, 9), ("prefill", 1, 40), ("prefill", 0, 30)])
def test_streaming_copy_that_never_comes_is_reported_and_recoverable(cuda_lib, call, quant, T):
    H, I, E, K = 512, 256, 16, 4
    lay = synth.LayerLayout(H, I, E, quant)
    blob = synth.make_layer_blob(lay, 0)
    sc = moe.allocate_moe_scratch(H, I, E, K, 64, flags=_lib.FLAG_SHORT_WAITS)
    layer = sc.prepare_layer(blob, lay.meta())
    x = torch.randn((T, H), generator=torch.Generator("cuda").manual_seed(T), device="cuda")
    run = sc.decode if call == "decode" else sc.prefill
    good = run(layer, x, x.clone()).clone()
    torch.cuda.synchronize()
    assert sc.poll_status() == _lib.OK
    sc.debug_expire_next_wait(0 if call == "decode" else 1)
    run(layer, x, x.clone())
    torch.cuda.synchronize()
    assert sc.poll_status() == _lib.TIMEOUT
    with pytest.raises(moe.LumenMoeError) as ei:
        run(layer, x, x.clone())
    assert ei.value.code == _lib.TIMEOUT
    sc.clear_status()
    again = run(layer, x, x.clone())
    torch.cuda.synchronize()
    assert sc.poll_status() == _lib.OK and torch.equal(again, good)


def test_expert_id_out_of_range_is_an_error_code_not_a_fault(cuda_lib):
    # caller-supplied routing (what an expert-parallel rank receives over the wire): an id >= E must
    # never index a table; the pair is dropped (expert 0, weight 0) and the context reports INVALID_ARG
    H, I, E, K, T = 256, 128, 8, 2, 50
    _, blob, sc, layer = _ctx(H, I, E, K, T)
    g = torch.Generator("cuda").manual_seed(5)
    x = torch.randn((T, H), generator=g, device="cuda")
    res = torch.randn((T, H), generator=g, device="cuda")
    ids = torch.randint(0, E, (T, K), generator=g, device="cuda", dtype=torch.int32)
    w = torch.rand((T, K), generator=g, device="cuda")
    ok = sc.prefill_routed(layer, x, ids, w, res).clone()
    torch.cuda.synchronize()
    assert sc.poll_status() == _lib.OK
    bad = ids.clone()
    bad[7, 1] = E + 3
    bad[20, 0] = -1                      # 0xffffffff as u32
    out = sc.prefill_routed(layer, x, bad, w, res)
    torch.cuda.synchronize()
    assert sc.poll_status() == _lib.INVALID_ARG
    # rows whose ids were valid are unaffected; the dropped pairs contribute nothing
    w0 = w.clone()
    w0[7, 1] = 0.0
    w0[20, 0] = 0.0
    fixed = ids.clone()
    fixed[7, 1] = 0
    fixed[20, 0] = 0
    sc.clear_status()
    ref = sc.prefill_routed(layer, x, fixed, w0, res)
    torch.cuda.synchronize()
    assert torch.equal(out, ref)
    assert not torch.equal(out, ok)


def test_ids_in_the_reference_stride_e_layout(cuda_lib):
    E, K, T = 64, 4, 9
    sc = moe.allocate_moe_scratch(256, 128, E, K, 16)
    lg = synth.uniform_logits(T, E, 11, tau=1.0)
    ids, _ = sc.topk_from_logits(lg)
    wide = sc.get_routing_ids_stride_e(T)
    o_ids, _ = oracle.topk_from_logits(lg.cpu().numpy(), K, 0)
    assert wide.shape == (T, E)
    assert np.array_equal(wide[:, :K], o_ids) and not wide[:, K:].any()
    assert np.array_equal(ids.cpu().numpy().astype(np.uint32), wide[:, :K])
    # the reference's host counting sort walks this buffer with stride E (cuda/moe.rs:2116-2121)
    r = sc.get_routing(T)
    _, cst, d2c, bounds = oracle.counting_sort(wide, E, K=K)
    assert np.array_equal(r["dst_to_col"], d2c) and np.array_equal(r["col_src_tok"], cst)
    assert np.array_equal(r["expert_bounds"], bounds)


def test_pointers_between_16_byte_boundaries_are_refused_where_kernels_need_them(cuda_lib):
    H, I, E, K, T = 512, 256, 16, 4, 3
    _, blob, sc, layer = _ctx(H, I, E, K, 64)
    one = _ctx(H, I, E, 1, 64)
    x, off = torch.randn((T, H), device="cuda"), torch.zeros(T * H + 1, device="cuda")[1:].view(T, H)
    gamma, gamma_off = torch.ones(H, device="cuda"), torch.ones(H + 1, device="cuda")[1:]
    ids = torch.zeros(200, device="cuda", dtype=torch.int32)
    rows16, out16 = torch.zeros((200, H), device="cuda"), torch.zeros(200 * H + 1, device="cuda", dtype=torch.float16)[1:]
    sc.route_only(layer, x)  # leaves the tables ep_prepare needs
    lib = _lib.lib()
    calls = [
        lambda: sc.decode(layer, off, x),
        lambda: sc.decode_fused_norm(layer, off, gamma, 1e-6),
        lambda: sc.decode_fused_norm(layer, x, gamma_off, 1e-6),
        lambda: sc.decode_fused_norm(layer, x, gamma, 1e-6, off),
        lambda: sc.stack_decode([layer], [gamma], off, 1e-6),
        lambda: sc.stack_decode([layer, layer], [gamma, gamma_off], x, 1e-6),
        lambda: sc.route_only(layer, off),
        lambda: moe.quantize(off.view(-1), 1),
        lambda: _lib.check(lib.lumen_moe_experts_routed_f16(one[2]._h, one[3]._h, rows16.data_ptr(), ids.data_ptr(), out16.data_ptr(), 200, 0, 0)),
        lambda: _lib.check(lib.lumen_moe_ep_prepare(sc._h, x.data_ptr(), 0, T, 4, out16.data_ptr(), ids.data_ptr(), ids.data_ptr(), 0)),
    ]
    for call in calls:
        with pytest.raises(moe.LumenMoeError) as ei:
            call()
        assert ei.value.code == _lib.INVALID_ARG and "16-byte" in str(ei.value)
    assert torch.isfinite(sc.decode(layer, x, off, off)).all() and sc.poll_status() == _lib.OK


@pytest.mark.parametrize("which", ["router_weight_off", "expert_gate_offs", "expert_up_offs", "expert_down_offs"])
@pytest.mark.parametrize("off", [2**64 - 64, 2**63, "one past the end"])
def test_layer_offsets_outside_the_blob_are_refused(cuda_lib, which, off):
    # an offset so large that offset + length wraps round must not pass for a small one
    H, I, E = 256, 128, 4
    lay = synth.LayerLayout(H, I, E, 1)
    blob = synth.make_layer_blob(lay, 0)
    sc = moe.allocate_moe_scratch(H, I, E, 2, 16)
    meta = lay.meta()
    value = off if isinstance(off, int) else blob.numel()
    if which == "router_weight_off":
        meta.router_weight_off = value // 4 * 4
    else:
        offs = list(getattr(meta, which))
        offs[2] = value
        setattr(meta, which, offs)
    with pytest.raises(moe.LumenMoeError) as ei:
        sc.prepare_layer(blob, meta)
    assert ei.value.code == _lib.INVALID_ARG
    sc.prepare_layer(blob, lay.meta())  # the context is none the worse


def test_unknown_config_flags_are_rejected(cuda_lib):
    with pytest.raises(moe.LumenMoeError):
        moe.allocate_moe_scratch(256, 128, 8, 2, 16, flags=0x10)


def test_contexts_on_two_devices_in_one_process(cuda_lib):
    # the shared-memory opt-in of a kernel is per device: a second GPU must get its own
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    H, I, E, K = 512, 256, 16, 4
    outs = []
    for dev in (0, 1):
        torch.cuda.set_device(dev)
        _, blob, sc, layer = _ctx(H, I, E, K, 300, device=dev)
        g = torch.Generator(f"cuda:{dev}").manual_seed(6)
        x = torch.randn((300, H), generator=g, device=f"cuda:{dev}")
        res = torch.zeros((300, H), device=f"cuda:{dev}")
        p = sc.prefill(layer, x, res)
        d16 = sc.decode(layer, x[:16].contiguous(), res[:16].contiguous())
        d2 = sc.decode(layer, x[:2].contiguous(), res[:2].contiguous())
        torch.cuda.synchronize()
        outs.append((p.cpu(), d16.cpu(), d2.cpu()))
    torch.cuda.set_device(0)
    for a, b in zip(*outs):
        assert torch.equal(a, b)
