"""The tcgen05 kernels on rings of few shared-memory stages (the tc_stages tuning, 2 to 8): with fewer stages than producer
warps, rings shorter and longer than a tile's k-blocks, several tiles and K splits per CTA."""
import numpy as np
import pytest
from gpu_util import run_linear
from linear_check import assert_close

from vai_b200 import nodes

pytestmark = pytest.mark.gpu


def _draw(M, K, N):
    rng = np.random.default_rng(M + 3 * K + 5 * N)
    return (rng.standard_normal((M, K)).astype(np.float32), (rng.standard_normal((N, K)) / np.sqrt(K)).astype(np.float32),
            rng.standard_normal(N).astype(np.float32))


@pytest.mark.parametrize("stages", [2, 3, 4])
@pytest.mark.parametrize("M,K,N,kernel,extra", [
    (300, 2056, 40000, nodes.KERNEL_TC_GEMM, dict(tc_pair=1)), (300, 2056, 520, nodes.KERNEL_TC_GEMM, dict(tc_pair=1, tc_splits=3)),
    (300, 1032, 9000, nodes.KERNEL_TC_GEMM, dict(tc_pair=0)), (24, 2056, 30000, nodes.KERNEL_TC_SKINNY, {}),
    (64, 4096, 520, nodes.KERNEL_TC_SKINNY, dict(tc_splits=5)), (64, 72, 20000, nodes.KERNEL_TC_SKINNY, {})])
def test_ring_depth(stages, M, K, N, kernel, extra, device):
    x, w, b = _draw(M, K, N)
    got, want, _ = run_linear(x, w, b, i_dtype="bf16", w_dtype="bf16", kernel=kernel, tuning=dict(tc_stages=stages, **extra))
    assert_close(got, want, (2e-4, 5e-5), f"{M}x{K}x{N} stages={stages} {extra}")     # fp32 sums of exact products


@pytest.mark.parametrize("stages", [2, 3])
@pytest.mark.parametrize("M,kernel", [(200, nodes.KERNEL_TC_GEMM), (40, nodes.KERNEL_TC_SKINNY)])
def test_ring_depth_gate(stages, M, kernel, device):
    x, w, b = _draw(M, 1544, 2 * 9000)
    got, want, _ = run_linear(x, w, b, w_dtype="f16", epilogue="SILU", gate_fuse=True, kernel=kernel, tuning=dict(tc_stages=stages))
    assert_close(got, want, (2e-4, 5e-5), f"gate M={M} stages={stages}")
