"""A Linear whose weight was written on its stream: by a norm just ahead of it, with other launches in between, and wired
from a node in a net.  The Linear kernels request their weights before the launch ahead has completed."""
import ctypes

import numpy as np
import pytest
import torch
from linear_check import assert_close

from vai_b200 import Dtype, NeuralNet, Tensor, _lib, nodes

pytestmark = pytest.mark.gpu
N, K = 6144, 2048            # 12.6 M elements: the norm takes longer than a dependent launch needs to arrive


def _normed(x):
    """RmsNorm of fp32 rows in float64, as stored in bf16."""
    y = x.double() / torch.sqrt((x.double() ** 2).mean(-1, keepdim=True) + 1e-5)
    return y.float().bfloat16().double()


@pytest.mark.parametrize("M", [1, 2, 6, 40, 200])
@pytest.mark.parametrize("between", [None, "norm", "topk"])
def test_norm_then_linear(M, between, device):
    lib, f32, bf16 = device.lib, int(Dtype.F32), int(Dtype.BF16)
    d = _lib.LinearDesc(M=M, N=N, K=K, i_dtype=bf16, w_dtype=bf16, o_dtype=f32, b_dtype=int(Dtype.NONE), scalar_scale=1.0)
    plan, info = ctypes.c_void_p(), _lib.LinearInfo()
    _lib.check(lib.vaicu_linear_plan_create(device.handle, ctypes.byref(d), ctypes.byref(plan)), "plan")
    _lib.check(lib.vaicu_linear_plan_info(plan, ctypes.byref(info)), "info")
    ws = torch.empty(max(info.workspace_bytes, 256), dtype=torch.uint8, device="cuda")
    w, out = torch.zeros(N, K, dtype=torch.bfloat16, device="cuda"), torch.empty(M, N, device="cuda")
    x, small, small_out = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(4, K, device="cuda"), torch.empty(4, K, device="cuda")
    pick, uniform = torch.zeros(4, dtype=torch.int32, device="cuda"), torch.full((1,), 0.5, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    for i in range(4):
        raw = torch.randn(N, K, device="cuda")
        _lib.check(lib.vaicu_rms_norm_run(device.handle, s, raw.data_ptr(), None, None, None, w.data_ptr(), N, K, f32, f32, bf16, 1e-5), "norm")
        if between == "norm":
            _lib.check(lib.vaicu_rms_norm_run(device.handle, s, small.data_ptr(), None, None, None, small_out.data_ptr(), 4, K, f32, f32, f32, 1e-5), "norm")
        elif between == "topk":
            _lib.check(lib.vaicu_topk_sample_run(s, small.data_ptr(), f32, 4, K, 8, 1.0, uniform.data_ptr(), None, pick.data_ptr()), "topk")
        _lib.check(lib.vaicu_linear_run(plan, s, x.data_ptr(), w.data_ptr(), None, None, out.data_ptr(), ws.data_ptr()), "linear")
        assert_close(w.float().cpu().numpy(), _normed(raw).cpu().numpy(), (2.0 ** -7, 1e-6), "the norm")       # one bf16 step
        want = (x.double() @ w.double().t()).cpu().numpy()                       # with the weights as they were stored
        assert_close(out.cpu().numpy(), want, (1e-4, 1e-3), f"M={M} between={between} call {i}")       # fp32 sums of 2048 products
    torch.cuda.synchronize()
    lib.vaicu_linear_plan_destroy(plan)


@pytest.mark.parametrize("M", [1, 6, 200])
def test_wired_norm(M, device):
    net = NeuralNet(w_default_dtype=Dtype.BF16)
    norm, lin = nodes.RmsNormNode(), nodes.LinearNode(in_dim=K, out_dim=N)
    norm.set_o_dtype(Dtype.BF16)
    net.input("x") - lin - net.output("y")
    net.input("w") - norm
    norm - "weight" / lin
    rng = np.random.default_rng(M)
    for i in range(3):
        x, raw = rng.standard_normal((M, K), dtype=np.float32), rng.standard_normal((N, K), dtype=np.float32)
        x = torch.from_numpy(x).bfloat16().float().numpy()
        got = net(x=Tensor.from_numpy(x), w=Tensor.from_numpy(raw)).to_numpy()
        # a weight at the edge of a bf16 rounding may fall on its other side, 2^-8 of up to 4, times an activation of up to 4:
        # four of them in one output.  Outputs are of the order of 45; a weight read too early is the last call's.
        assert_close(got, (torch.from_numpy(x).double() @ _normed(torch.from_numpy(raw)).t()).numpy(), (1e-4, 0.25), f"M={M} call {i}")


@pytest.mark.parametrize("M,argmax", [(1, False), (1, True), (6, False), (40, False), (200, False)])
def test_wired_linear(M, argmax, device):
    """The weight is another Linear's output: that kernel lets its successor start early."""
    net = NeuralNet(w_default_dtype=Dtype.BF16)
    inner, lin = nodes.LinearNode(in_dim=K, out_dim=K), nodes.LinearNode(in_dim=K, out_dim=N)
    inner.set_o_dtype(Dtype.BF16)
    rng = np.random.default_rng(M)
    inner["weight"] = Tensor.from_numpy(np.eye(K, dtype=np.float32)[::-1].copy(), dtype=Dtype.BF16)      # reverses the columns: exact
    if argmax:
        net.input("x") - lin - nodes.ArgmaxNode() - net.output("y")
    else:
        net.input("x") - lin - net.output("y")
    net.input("w") - inner
    inner - "weight" / lin
    for i in range(3):
        x = torch.from_numpy(rng.standard_normal((M, K), dtype=np.float32)).bfloat16()
        raw = torch.from_numpy(rng.standard_normal((N, K), dtype=np.float32)).bfloat16()
        got = net(x=Tensor.from_numpy(x.float().numpy()), w=Tensor.from_numpy(raw.float().numpy()))
        want = x.double() @ raw.double().flip(1).t()
        if argmax:
            np.testing.assert_array_equal(got.to_u32().reshape(-1), want.argmax(-1).numpy())
        else:
            assert_close(got.to_numpy(), want.numpy(), (1e-4, 1e-3), f"M={M} call {i}")      # fp32 sums of exact products
