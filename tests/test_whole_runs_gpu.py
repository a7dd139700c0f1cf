"""Runs with several destinations (scatter, broadcast, reduce-scatter) on plans whose K the library splits by its own choice:
the epilogue must see finished sums, so these runs keep K whole; a split that the caller asked for is refused."""
import ctypes

import pytest
import torch
from linear_check import assert_close

from vai_b200 import Dtype, _lib

pytestmark = pytest.mark.gpu
UNSUPPORTED = 2


class Plan:
    def __init__(self, device, M, N, K, **fields):
        tuning = fields.pop("tuning", {})
        self.lib = device.lib
        d = _lib.LinearDesc(M=M, N=N, K=K, i_dtype=int(Dtype.BF16), w_dtype=int(Dtype.BF16), o_dtype=int(Dtype.F32), b_dtype=int(Dtype.NONE),
                            scalar_scale=1.0, **fields)
        t = _lib.LinearTuning(**tuning)
        self.h, self.info = ctypes.c_void_p(), _lib.LinearInfo()
        _lib.check(self.lib.vaicu_linear_plan_create_tuned(device.handle, ctypes.byref(d), ctypes.byref(t), ctypes.byref(self.h)), "plan")
        _lib.check(self.lib.vaicu_linear_plan_info(self.h, ctypes.byref(self.info)), "info")
        g = torch.Generator(device="cuda").manual_seed(M + N + K)
        self.x, self.w = (torch.randn(s, K, device="cuda", generator=g).bfloat16() for s in (M, N))
        self.ws = torch.empty(max(self.info.workspace_bytes, 256), dtype=torch.uint8, device="cuda")
        self.want = (self.x.double() @ self.w.double().t()).cpu().numpy()
        self.s = torch.cuda.current_stream().cuda_stream

    def __del__(self):
        self.lib.vaicu_linear_plan_destroy(self.h)


def _ptrs(ts):
    return (ctypes.c_void_p * len(ts))(*[t.data_ptr() for t in ts])


@pytest.mark.parametrize("M,K,N", [(130, 2560, 3072), (334, 2048, 8192), (24, 3072, 3072), (16, 4096, 2560)])
def test_whole_runs_of_split_plans(M, K, N, device):
    p = Plan(device, M, N, K)
    tol = (1e-4, 2e-3)                  # fp32 sums of up to 4096 products of N(0, 1) values
    outs = [torch.zeros(M, N + 64, device="cuda") for _ in range(2)]
    _lib.check(p.lib.vaicu_linear_run_scatter(p.h, p.s, p.x.data_ptr(), p.w.data_ptr(), None, _ptrs(outs), 2, N + 64, 64, p.ws.data_ptr()), "scatter")
    for o in outs:
        assert_close(o[:, 64:].cpu().numpy(), p.want, tol, "scatter")
        assert not o[:, :64].any()
    outs = [torch.zeros(M, N, device="cuda") for _ in range(3)]
    _lib.check(p.lib.vaicu_linear_run_broadcast(p.h, p.s, p.x.data_ptr(), p.w.data_ptr(), None, None, _ptrs(outs), 3, p.ws.data_ptr()), "broadcast")
    for o in outs:
        assert_close(o.cpu().numpy(), p.want, tol, "broadcast")
    parts = [torch.zeros(2, M // 2, N, device="cuda") for _ in range(2)]
    _lib.check(p.lib.vaicu_linear_run_reduce_scatter(p.h, p.s, p.x.data_ptr(), p.w.data_ptr(), _ptrs(parts), 2, 1, p.ws.data_ptr()), "reduce_scatter")
    assert_close(torch.cat([t[1] for t in parts]).cpu().numpy(), p.want, tol, "reduce_scatter")
    assert not any(t[0].any() for t in parts)
    kernel, vec = ctypes.c_int(), ctypes.c_int()
    _lib.check(p.lib.vaicu_linear_plan_last_run(p.h, ctypes.byref(kernel), ctypes.byref(vec)), "last_run")
    assert kernel.value == p.info.kernel
    out = torch.zeros(M, N, device="cuda")             # and the plan itself is as it was
    _lib.check(p.lib.vaicu_linear_run(p.h, p.s, p.x.data_ptr(), p.w.data_ptr(), None, None, out.data_ptr(), p.ws.data_ptr()), "run")
    assert_close(out.cpu().numpy(), p.want, tol, "run")


@pytest.mark.parametrize("M,K,N,fields", [(130, 4096, 3072, dict(split_size=1024)), (130, 4096, 3072, dict(tuning=dict(tc_splits=2))),
                                          (24, 4096, 3072, dict(tuning=dict(tc_splits=4))), (130, 4096, 64, {}), (24, 4096, 512, {})])
def test_splits_that_stay_refused(M, K, N, fields, device):
    p = Plan(device, M, N, K, **fields)
    out = torch.zeros(M, N, device="cuda")
    assert p.info.split_count > 1
    assert p.lib.vaicu_linear_run_scatter(p.h, p.s, p.x.data_ptr(), p.w.data_ptr(), None, _ptrs([out]), 1, N, 0, p.ws.data_ptr()) == UNSUPPORTED
    assert p.lib.vaicu_linear_run_broadcast(p.h, p.s, p.x.data_ptr(), p.w.data_ptr(), None, None, _ptrs([out]), 1, p.ws.data_ptr()) == UNSUPPORTED
    assert p.lib.vaicu_linear_run_reduce_scatter(p.h, p.s, p.x.data_ptr(), p.w.data_ptr(), _ptrs([out]), 1, 0, p.ws.data_ptr()) == UNSUPPORTED
