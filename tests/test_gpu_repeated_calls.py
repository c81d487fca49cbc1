"""Calls that are made over and over are replayed from a graph: the results must follow the inputs all the same."""
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


@pytest.mark.parametrize("where", ["device", "host"])
@pytest.mark.parametrize("m", [1, 5, 200])
def test_repeated_call_follows_its_inputs(torch, oracle, m, where):
    """One row (fused quantize), a batch and a prefill on the same buffers, with new activations in place each time and, in
    between, a call that makes the library's workspace and arena grow."""
    import weft_b200 as weft
    from weft_b200.kernels import mul_mat
    from weft_b200.runtime import Buffer

    n, k = 96, 1024
    rng = np.random.default_rng(m)
    packed = weights(oracle.Q4_K, rng, n, k)
    kernel = weft.compile(mul_mat.production_mul_mat_q4_k_staged)
    w = Buffer(torch.from_numpy(packed).cuda(), shape=(n, k), encoding="Q4_K")
    x, xq, y = np.zeros((m, k), np.float32), np.zeros((m, oracle.row_bytes(oracle.Q8_K, k)), np.uint8), np.zeros((m, n), np.float32)
    if where == "device":
        x, xq, y = (torch.from_numpy(a).cuda() for a in (x, xq, y))
    args = (w, Buffer(x), Buffer(xq, shape=(m, k), encoding="Q8_K"), Buffer(y))
    host = (lambda a: a.cpu().numpy()) if where == "device" else (lambda a: a)
    for call in range(8):
        fresh = activations(rng, m, k) * (1 + call)
        if where == "device":
            x.copy_(torch.from_numpy(fresh))
            torch.cuda.synchronize()
        else:
            x[:] = fresh
        kernel(*args)
        want, want_xq = oracle.mul_mat(oracle.Q4_K, packed, fresh, n, k, m, rule=1)
        assert np.array_equal(host(xq), want_xq), call
        assert rel_l2(host(y), want) <= 1e-5, call
        if call == 5:
            big = 700 * m
            kernel(w, torch.zeros((big, k), device="cuda"), Buffer(torch.zeros((big, xq.shape[1]), dtype=torch.uint8, device="cuda"), shape=(big, k), encoding="Q8_K"),
                   np.zeros((big, n), np.float32))
