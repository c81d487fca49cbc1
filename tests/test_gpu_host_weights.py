"""Weights in ordinary host memory, other ones at each call: the kernels fetch their first weights ahead of their wait for the
kernel before them, so the copy that brings host weights must be complete by then.  24 calls on the same buffers: the last
seven are replayed from a graph.  Bound: 1e-5 relative L2 (exact integer sums, another order of the fp32 additions)."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import activations, rel_l2, weights

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch

    if not torch.cuda.is_available():
        pytest.fail("these tests need a CUDA device; there is no CPU fallback to test")
    return torch


@pytest.mark.parametrize("name", ["Q4_K", "Q6_K", "Q8_0"])
@pytest.mark.parametrize("pinned", [False, True])
def test_weights_of_this_call(torch, oracle, name, pinned):
    """One token row, activations on the device: the weights are the last argument on its way when the GEMV is launched."""
    import weft_b200 as weft
    from weft_b200.kernels import mul_mat
    from weft_b200.runtime import Buffer

    n, k, act = 96, 1024, "Q8_0" if name == "Q8_0" else "Q8_K"
    fmt, act_fmt = getattr(oracle, name), getattr(oracle, act)
    rng = np.random.default_rng(n)
    kernel = weft.compile(getattr(mul_mat, f"production_mul_mat_{name.lower()}_decode"))
    x = activations(rng, 1, k)
    held = torch.zeros((n, oracle.row_bytes(fmt, k)), dtype=torch.uint8, pin_memory=pinned).numpy()
    xq = torch.zeros((1, oracle.row_bytes(act_fmt, k)), dtype=torch.uint8, device="cuda")
    y = torch.zeros((1, n), device="cuda")
    args = (Buffer(held, shape=(n, k), encoding=name), Buffer(torch.from_numpy(x).cuda()), Buffer(xq, shape=(1, k), encoding=act), Buffer(y))
    for call in range(24):
        held[:] = weights(fmt, rng, n, k)
        kernel(*args)
        want, _ = oracle.mul_mat(fmt, held.copy(), x, n, k, 1, rule=1)
        assert rel_l2(y.cpu().numpy(), want) <= 1e-5, call


def test_interleaved_weights_behind_a_large_copy(torch, oracle):
    """Everything on the host and X too large for a copy kernel: the copy of the weights comes last."""
    import weft_b200 as weft
    from weft_b200.kernels import mul_mat
    from weft_b200.runtime import Buffer

    m, n, k = 128, 64, 1024
    rng = np.random.default_rng(m)
    kernel = weft.compile(mul_mat.production_mul_mat_q4_k_persistent)
    x, held = activations(rng, m, k), np.zeros((n, k // 256 * 144), np.uint8)
    xq, y = np.zeros((m, oracle.row_bytes(oracle.Q8_K, k)), np.uint8), np.zeros((m, n), np.float32)
    for call in range(24):
        w = weights(oracle.Q4_K, rng, n, k)
        held[:] = oracle.interleave(oracle.Q4_K, w, k).reshape(held.shape)
        kernel(Buffer(held, shape=(n, k), encoding="Q4K_I[16]"), Buffer(x), Buffer(xq, shape=(m, k), encoding="Q8_K"), Buffer(y))
        want, _ = oracle.mul_mat(oracle.Q4_K, w, x, n, k, m, rule=1)
        assert rel_l2(y, want) <= 1e-5, call
