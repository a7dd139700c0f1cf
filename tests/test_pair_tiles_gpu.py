"""The CTA-pair kernel at every width its cost model picks from, whole and split along K: ragged rows and columns, K tails,
fewer k-blocks than stages, finished tiles stored through shared memory or directly, partial sums as whole or single
elements (N % 4 != 0), residuals one chunk ahead."""
import ctypes

import numpy as np
import pytest
from gpu_util import out_tol, run_linear
from linear_check import assert_close

from vai_b200 import Dtype, _lib, nodes

pytestmark = pytest.mark.gpu


def _draw(M, K, N):
    rng = np.random.default_rng(M + 3 * K + 5 * N)
    return (rng.standard_normal((M, K)).astype(np.float32), (rng.standard_normal((N, K)) / np.sqrt(K)).astype(np.float32),
            rng.standard_normal(N).astype(np.float32), rng.standard_normal((M, N)).astype(np.float32))


@pytest.mark.parametrize("bn", [64, 96, 128, 192, 256])
@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("M,K,N", [(129, 776, 768), (333, 1160, 530), (600, 200, 1000)])
@pytest.mark.parametrize("o_dtype", ["f32", "bf16"])
def test_pair_widths(bn, splits, M, K, N, o_dtype, device):
    x, w, b, r = _draw(M, K, N)
    got, want, node = run_linear(x, w, b, r, i_dtype="bf16", w_dtype="bf16", o_dtype=o_dtype, epilogue="SILU", kernel=nodes.KERNEL_TC_GEMM,
                                 tuning=dict(tc_pair=1, tc_bn=bn, tc_splits=splits))
    assert node.info.tile_n == bn
    assert_close(got, want, out_tol(o_dtype, 2e-4, 5e-5), f"{M}x{K}x{N} bn={bn} splits={splits}")


@pytest.mark.parametrize("bn", [64, 96, 192, 256])
@pytest.mark.parametrize("splits", [1, 2])
@pytest.mark.parametrize("H", [520, 333])
def test_pair_widths_gate(bn, splits, H, device):
    x, w, b, _ = _draw(200, 520, 2 * H)
    got, want, _ = run_linear(x, w, b, w_dtype="f16", epilogue="GELU_TANH", gate_fuse=True, kernel=nodes.KERNEL_TC_GEMM,
                              tuning=dict(tc_pair=1, tc_bn=bn, tc_splits=splits))
    assert_close(got, want, (2e-4, 5e-5), f"gate H={H} bn={bn} splits={splits}")


@pytest.mark.parametrize("M,K,N", [(160, 8192, 512), (333, 768, 768), (700, 2048, 520), (257, 64, 4096), (17, 3072, 3072), (24, 4096, 2561)])
def test_chosen_tiles(M, K, N, device):
    """What the planner picks by itself, against float64."""
    x, w, b, r = _draw(M, K, N)
    got, want, node = run_linear(x, w, b, r, w_dtype="bf16")
    assert node.info.kernel == (nodes.KERNEL_TC_GEMM if M > 128 else nodes.KERNEL_TC_SKINNY)
    assert_close(got, want, (2e-4, 5e-5), f"{M}x{K}x{N}")


@pytest.mark.parametrize("M,K,N,gate,widest", [(40000, 768, 64, False, 64), (40000, 768, 100, False, 128), (20000, 2048, 300, False, 192),
                                               (40000, 768, 768, False, 256), (8192, 768, 2048, False, 256), (40000, 768, 2 * 40, True, 64)])
def test_tall_layers_do_not_compute_padding(M, K, N, gate, widest, device):
    """Many rounds of tiles, few columns: the widest tile only where the output fills it."""
    d = _lib.LinearDesc(M=M, N=N, K=K, i_dtype=int(Dtype.BF16), w_dtype=int(Dtype.BF16), o_dtype=int(Dtype.BF16), b_dtype=int(Dtype.NONE),
                        scalar_scale=1.0, gate_fuse=int(gate))
    plan, info = ctypes.c_void_p(), _lib.LinearInfo()
    _lib.check(device.lib.vaicu_linear_plan_create(device.handle, ctypes.byref(d), ctypes.byref(plan)), "plan")
    _lib.check(device.lib.vaicu_linear_plan_info(plan, ctypes.byref(info)), "info")
    assert info.tile_n == widest
    device.lib.vaicu_linear_plan_destroy(plan)


@pytest.mark.parametrize("M,N", [(9480 * 2, 300), (40000, 64)])
def test_tall_layers(M, N, device):
    x, w, b, _ = _draw(M, 72, N)
    got, want, _ = run_linear(x, w, b, i_dtype="bf16", w_dtype="bf16", o_dtype="bf16")
    assert_close(got, want, out_tol("bf16", 2e-4, 5e-5), f"{M}x72x{N}")


@pytest.mark.parametrize("bn", [64, 128, 192, 256])
@pytest.mark.parametrize("M,N,gate", [(129, 333, False), (300, 1001, False), (520, 2 * 333, True), (257, 129, False)])
def test_rows_of_odd_width_in_fp32(bn, M, N, gate, device):
    """Output rows that begin at any fp32 element go through shared memory too, a store instruction per row."""
    x, w, b, r = _draw(M, 200, N)
    got, want, node = run_linear(x, w, b, None if gate else r, i_dtype="bf16", w_dtype="bf16", epilogue="GELU" if gate else "SILU", gate_fuse=gate,
                                 kernel=nodes.KERNEL_TC_GEMM, tuning=dict(tc_pair=1, tc_bn=bn, tc_splits=1))
    assert_close(got, want, (2e-4, 5e-5), f"{M}x200x{N} bn={bn}")
