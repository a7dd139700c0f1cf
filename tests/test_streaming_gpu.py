"""The streaming decode forms (gemv_stream.cu for one row, skinny_stream.cu for 5 to 8) at the sizes where their
geometry can go wrong: K that fills no vector round, one that needs several warps or several register
loads of activations, fewer columns than blocks, ranges that end inside a stage, more columns than one fold holds."""
import ctypes

import numpy as np
import pytest
import torch
from gpu_util import out_tol, run_linear, seen
from linear_check import assert_close

from oracle import linear_oracle as orc
from vai_b200 import Dtype, Epilogue, NeuralNet, Tensor, _lib, nodes

pytestmark = pytest.mark.gpu


def _draw(M, K, N, residual=True):
    rng = np.random.default_rng(M * 7919 + K * 31 + N)
    return (rng.standard_normal((M, K)).astype(np.float32), (rng.standard_normal((N, K)) / np.sqrt(K)).astype(np.float32),
            rng.standard_normal(N).astype(np.float32), rng.standard_normal((M, N)).astype(np.float32) if residual else None)


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("K,N", [(8, 3), (200, 147), (520, 149), (768, 768), (1032, 300), (2560, 611), (4096, 160), (4104, 152),
                                 (8192, 320), (12288, 150), (64, 70001)])
@pytest.mark.parametrize("dt", [("f32", "f16", "f32"), ("bf16", "bf16", "bf16")])
def test_streaming_plain(M, K, N, dt, device):
    x, w, b, r = _draw(M, K, N)
    got, want, node = run_linear(x, w, b, r, i_dtype=dt[0], w_dtype=dt[1], o_dtype=dt[2], epilogue="GELU", scalar_scale=0.5)
    assert node.info.kernel == (nodes.KERNEL_GEMV if M <= 4 else nodes.KERNEL_TC_SKINNY)
    assert node.info.launches == 1 or M > 4
    # fp32 sums; the error-function polynomial of the GELU is good to 1.5e-7 of its argument
    assert_close(got, want, out_tol(dt[2]), f"{M}x{K}x{N} {dt}")


@pytest.mark.parametrize("M", [1, 3, 4, 6])
@pytest.mark.parametrize("K,H", [(8, 5), (768, 1500), (2048, 149), (8192, 75), (520, 20000)])
@pytest.mark.parametrize("w_dtype", ["bf16", "f16"])
def test_streaming_gate(M, K, H, w_dtype, device):
    x, w, b, _ = _draw(M, K, 2 * H, residual=False)
    for ep in ("SILU", "GELU_TANH"):
        got, want, _ = run_linear(x, w, b, w_dtype=w_dtype, epilogue=ep, gate_fuse=True)
        assert_close(got, want, (1e-4, 1e-5), f"gate {ep} {M}x{K}x{H} {w_dtype}")


@pytest.mark.parametrize("M", [1, 3, 4, 8])
@pytest.mark.parametrize("K,widths", [(768, (128, 256, 128)), (2560, (2048, 1024, 1024)), (520, (128, 128))])
@pytest.mark.parametrize("io", ["f32", "bf16"])
def test_streaming_group(M, K, widths, io, device):
    """Sibling Linears of one input in one launch: ranges and stages that straddle the members."""
    _group(M, K, widths, io, 1)


@pytest.mark.parametrize("K,widths,tuning,launches", [(4096, (8192, 8192), None, 2), (2560, (1024, 1024), dict(tc_splits=1), 2),
                                                      (8200, (256, 128), None, 2), (4096, (8192, 4096), None, 1)])
def test_group_of_eight_rows_counts_its_launches(K, widths, tuning, launches, device):
    """GEMM and fold where the members together are too large for one launch, too deep, or tuned."""
    _group(8, K, widths, "bf16", launches, tuning)


def _group(M, K, widths, io, launches, tuning=None):
    rng = np.random.default_rng(K + M)
    x = rng.standard_normal((M, K)).astype(np.float32)
    ws = [(rng.standard_normal((n, K)) / np.sqrt(K)).astype(np.float32) for n in widths]
    dt = Dtype.BF16 if io == "bf16" else Dtype.F32
    net = NeuralNet(w_default_dtype=Dtype.BF16, o_default_dtype=dt, guard_bytes=512)
    src = net.input("x")
    for i, w in enumerate(ws):
        lin = nodes.LinearNode(in_dim=K, out_dim=w.shape[0], tuning=tuning)
        lin["weight"] = Tensor.from_numpy(w, dtype=Dtype.BF16)
        src - lin - net.output(f"y{i}")
    out = net(Tensor.from_numpy(x, dtype=dt))
    assert next(iter(net._recordings.values())).kernel_launches == launches
    net.pool.check_guards()
    xs = x if M <= 4 and io == "f32" else seen(x, Dtype.BF16)
    for i, w in enumerate(ws):
        assert_close(out[f"y{i}"].to_numpy(), orc.linear_f64(xs, seen(w, Dtype.BF16)), out_tol(io), f"member {i}")


@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("M", [5, 8])
def test_unaligned_fp32_activations_of_five_to_eight_rows(M, grouped, device):
    """Activations at any fp32 element: the same launch and the same bits as aligned ones, without a workspace."""
    K, widths, lib = 2056, (256, 384), device.lib
    g = torch.Generator(device="cuda").manual_seed(M)
    held = torch.randn(M * K + 4, device="cuda", generator=g)
    x = held[1:1 + M * K]
    same = x.clone()
    plans, ws, outs = [], [], []
    for n in widths:
        d = _lib.LinearDesc(M=M, N=n, K=K, i_dtype=int(Dtype.F32), w_dtype=int(Dtype.BF16), o_dtype=int(Dtype.F32), b_dtype=int(Dtype.NONE),
                            scalar_scale=1.0)
        h, info = ctypes.c_void_p(), _lib.LinearInfo()
        _lib.check(lib.vaicu_linear_plan_create(device.handle, ctypes.byref(d), ctypes.byref(h)), "plan")
        _lib.check(lib.vaicu_linear_plan_info(h, ctypes.byref(info)), "info")
        plans.append(h)
        ws.append(torch.randn(n, K, device="cuda", generator=g).bfloat16())
        outs.append([torch.zeros(M, n, device="cuda") for _ in range(2)])
        work = torch.empty(max(info.workspace_bytes, 256), dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    for k, act in enumerate((x, same)):
        if grouped:
            need = ctypes.c_size_t(1)
            arr = (ctypes.c_void_p * 2)(*plans)
            _lib.check(lib.vaicu_linear_group_workspace_bytes(arr, 2, ctypes.byref(need)), "group")
            assert need.value == 0
            _lib.check(lib.vaicu_linear_run_group(arr, 2, s, act.data_ptr(), (ctypes.c_void_p * 2)(*[w.data_ptr() for w in ws]),
                                                  (ctypes.c_void_p * 2)(*[o[k].data_ptr() for o in outs]), None), "run_group")
        else:
            for h, w, o in zip(plans, ws, outs):
                _lib.check(lib.vaicu_linear_run(h, s, act.data_ptr(), w.data_ptr(), None, None, o[k].data_ptr(), work.data_ptr()), "run")
    for w, o in zip(ws, outs):
        assert torch.equal(o[0], o[1])
        want = same.reshape(M, K).bfloat16().double() @ w.double().t()
        assert_close(o[0].cpu().numpy(), want.cpu().numpy(), (1e-4, 1e-3), "unaligned")
    for h in plans:
        lib.vaicu_linear_plan_destroy(h)


@pytest.mark.parametrize("M", [1, 2, 4])
@pytest.mark.parametrize("N", [5, 149, 70001])
def test_streaming_argmax(M, N, device):
    """The Argmax that shares the launch: equal logits in different blocks, the lower index wins."""
    rng = np.random.default_rng(N + M)
    K = 264
    x = np.abs(rng.standard_normal((M, K))).astype(np.float32)
    w = (rng.standard_normal((N, K)) * 0.01).astype(np.float32)
    best = sorted({N // 3, N - 1})
    w[best] = 1.0
    net = NeuralNet(w_default_dtype=Dtype.F16)
    lin = nodes.LinearNode(in_dim=K, out_dim=N)
    lin["weight"] = Tensor.from_numpy(w, dtype=Dtype.F16)
    net.input("x") - lin - nodes.ArgmaxNode() - net.output("token")
    for _ in range(2):
        np.testing.assert_array_equal(net(Tensor.from_numpy(x)).to_u32().reshape(-1), np.full(M, best[0], np.uint32))


def test_streaming_epilogues_and_orders(device):
    x, w, b, r = _draw(7, 776, 333)
    for M in (1, 2, 7):
        for ep in Epilogue:
            got, want, _ = run_linear(x[:M].copy(), w, b, r[:M].copy(), w_dtype="bf16", epilogue=ep.name,
                                      residual_order="BEFORE_EPILOGUE", scalar_scale=0.25)
            assert_close(got, want, (1e-4, 1e-5), f"{ep.name} M={M}")


@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("kernel", [nodes.KERNEL_AUTO, nodes.KERNEL_GEMV])
@pytest.mark.parametrize("dt", [Dtype.F16, Dtype.BF16])
def test_fused_argmax_stores_the_logits_of_a_run(M, kernel, dt, device):
    """vaicu_linear_run_argmax gives what vaicu_linear_run and an Argmax give: the same logits, to the bit, on the plan's kernel."""
    K, N, lib = 2560, 3000, device.lib
    g = torch.Generator(device="cuda").manual_seed(M)
    tdt = torch.float16 if dt == Dtype.F16 else torch.bfloat16
    x, w = (torch.randn(s, K, device="cuda", generator=g).to(tdt) for s in (M, N))
    d = _lib.LinearDesc(M=M, N=N, K=K, i_dtype=int(dt), w_dtype=int(dt), o_dtype=int(dt), b_dtype=int(Dtype.NONE), scalar_scale=1.0)
    plan, need = ctypes.c_void_p(), ctypes.c_size_t()
    tuning = _lib.LinearTuning(kernel=kernel)
    _lib.check(lib.vaicu_linear_plan_create_tuned(device.handle, ctypes.byref(d), ctypes.byref(tuning), ctypes.byref(plan)), "plan")
    _lib.check(lib.vaicu_linear_argmax_workspace_bytes(plan, ctypes.byref(need)), "workspace")
    ws, pick = torch.zeros(need.value, dtype=torch.uint8, device="cuda"), torch.zeros(M, dtype=torch.int32, device="cuda")
    alone, fused = torch.zeros(M, N, dtype=tdt, device="cuda"), torch.zeros(M, N, dtype=tdt, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    _lib.check(lib.vaicu_linear_run(plan, s, x.data_ptr(), w.data_ptr(), None, None, alone.data_ptr(), None), "run")
    _lib.check(lib.vaicu_linear_run_argmax(plan, s, x.data_ptr(), w.data_ptr(), None, None, fused.data_ptr(), ws.data_ptr(), 0, None,
                                           pick.data_ptr()), "run_argmax")
    assert torch.equal(alone, fused)
    lib.vaicu_linear_plan_destroy(plan)


@pytest.mark.parametrize("K,N,gate,streamed", [
    (2048, 8192, False, True), (2048, 148 * 96, False, True), (2048, 148 * 96 + 1, False, False), (1536, 148 * 96 + 1, False, True),
    (768, 148 * 112 + 1, False, False), (2048, 128256, False, False), (64, 16384, False, False), (2048, 16384, True, True),
    (2048, 148 * 112 + 2, True, False), (2056, 148 * 96 + 2, True, False), (8192, 2048, False, True), (8192, 148 * 16 + 1, False, False), (8192, 148 * 7, False, False),
    (8200, 2048, False, False), (12288, 300, False, False)])
def test_five_to_eight_rows_choice(K, N, gate, streamed, device):
    """Which layers of 5 to 8 rows take the one-launch form: fp32 activations, so the tcgen05 kernel has a cast ahead of it."""
    d = _lib.LinearDesc(M=8, N=N, K=K, i_dtype=int(Dtype.F32), w_dtype=int(Dtype.BF16), o_dtype=int(Dtype.F32), b_dtype=int(Dtype.NONE),
                        scalar_scale=1.0, gate_fuse=int(gate))
    plan, info = ctypes.c_void_p(), _lib.LinearInfo()
    _lib.check(device.lib.vaicu_linear_plan_create(device.handle, ctypes.byref(d), ctypes.byref(plan)), "plan")
    _lib.check(device.lib.vaicu_linear_plan_info(plan, ctypes.byref(info)), "info")
    assert (info.launches == 1) == streamed
    device.lib.vaicu_linear_plan_destroy(plan)


@pytest.mark.parametrize("M", [5, 8])
@pytest.mark.parametrize("K,N", [(1536, 148 * 112), (1536, 148 * 112 + 1), (8192, 148 * 16), (8192, 148 * 16 + 8), (4096, 14200)])
def test_five_to_eight_rows_on_both_sides_of_the_choice(M, K, N, device):
    x, w, b, r = _draw(M, K, N)
    got, want, _ = run_linear(x, w, b, r, w_dtype="bf16")
    assert_close(got, want, (1e-4, 1e-5), f"{M}x{K}x{N}")


@pytest.mark.parametrize("K,N,w,streamed", [
    (200, 768, "bf16", True), (200, 9000, "bf16", False), (568, 9000, "bf16", False), (576, 9000, "bf16", True), (768, 90000, "bf16", True), (768, 93000, "bf16", False), (8192, 8192, "bf16", True),
    (8200, 9000, "bf16", False), (400, 32768, "f32", True), (280, 32768, "f32", False), (16392, 3000, "bf16", False)])
def test_one_row_choice(K, N, w, streamed, device):
    """Which layers of one row stream: the block count shows in the workspace of the fused Argmax (8 bytes per block)."""
    d = _lib.LinearDesc(M=1, N=N, K=K, i_dtype=int(Dtype.F32), w_dtype=int(Dtype.BF16 if w == "bf16" else Dtype.F32), o_dtype=int(Dtype.F32),
                        b_dtype=int(Dtype.NONE), scalar_scale=1.0)
    plan, need, sms = ctypes.c_void_p(), ctypes.c_size_t(), ctypes.c_int()
    _lib.check(device.lib.vaicu_device_sm_count(device.handle, ctypes.byref(sms)), "sm_count")
    _lib.check(device.lib.vaicu_linear_plan_create(device.handle, ctypes.byref(d), ctypes.byref(plan)), "plan")
    _lib.check(device.lib.vaicu_linear_argmax_workspace_bytes(plan, ctypes.byref(need)), "workspace")
    assert (need.value == 256 + (sms.value * 8 + 255) // 256 * 256) == streamed
    device.lib.vaicu_linear_plan_destroy(plan)


@pytest.mark.parametrize("K,N,w", [(200, 148 * 16, "bf16"), (200, 148 * 16 + 1, "bf16"), (280, 32768, "f32"), (8200, 9000, "bf16")])
def test_one_row_on_both_sides_of_the_choice(K, N, w, device):
    x, wt, b, r = _draw(1, K, N)
    got, want, _ = run_linear(x, wt, b, r, w_dtype=w)
    assert_close(got, want, (1e-4, 1e-5), f"1x{K}x{N}")
