"""Top-k selection where its bound is least selective: winners crowded in one thread's or one slice's columns (more
entries reach the bound than the rank step keeps), fewer candidates than k, equal logits, infinities and NaN."""
import numpy as np
import pytest

from oracle import linear_oracle as orc
from vai_b200 import NeuralNet, Tensor, nodes

pytestmark = pytest.mark.gpu
LOW = np.float32(-3.4028235e38)


def _rows(N):
    rng = np.random.default_rng(N)
    base = rng.standard_normal(N).astype(np.float32)
    few = np.full(N, -np.inf, np.float32)
    few[[1, N // 2, N - 1]] = [0.5, 2.0, -1.0]
    mixed = base.copy()
    mixed[::3], mixed[5], mixed[7] = np.nan, 9.0, -np.inf
    strided = base.copy()
    strided[3 % 256::256] += 50.0                     # every winner in the columns of one thread per block
    zeros = np.zeros(N, np.float32)
    zeros[1::2] = -0.0
    return {"descending": np.sort(base)[::-1].copy(), "ascending": np.sort(base), "few": few, "mixed": mixed,
            "strided": strided, "zeros": zeros, "lowest": np.full(N, LOW, np.float32)}


@pytest.mark.parametrize("N", [33, 2048, 2049, 30000, 300001])
@pytest.mark.parametrize("k", [1, 40, 128])
def test_topk_bound(N, k, device):
    net = NeuralNet()
    pick = nodes.TopKSamplingNode(k=k, temperature=1.0)
    net.input("x") - pick - net.output("token")
    for name, row in _rows(N).items():
        for u in (0.0, 0.3, 0.999):
            pick.set_uniform(u)
            got = net(Tensor.from_numpy(row[None, :])).to_u32()
            np.testing.assert_array_equal(got, orc.topk_sample_c(row[None, :], k, 1.0, u), err_msg=f"{name} u={u}")
