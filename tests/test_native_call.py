"""The native call path takes exactly the calls that pass every check of the Python path, and leaves the rest to it."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest


@pytest.fixture(scope="module")
def plan_and_calls():
    from weft_b200.build import ensure_built
    from weft_b200.runtime import Buffer

    ensure_built()
    from weft_b200._pycall import Plan

    calls = []
    signature = ctypes.CFUNCTYPE(ctypes.c_int, *[ctypes.c_uint64] * 7)

    def record(*arguments):
        calls.append(arguments)
        return 0

    symbol = signature(record)
    # production_mul_mat_q4_k_decode: W (N, K), X (M, K), Xq (M, K), Y (M, N); extents N, K, M
    parameters = [("Q4_K", (0, 1), 256, 144, 2, 0, False), ("dense.f32", (2, 1), 1, 4, 4, 0, False), ("Q8_K", (2, 1), 256, 292, 4, 1, True),
                  ("dense.f32", (2, 0), 1, 4, 4, 2, True)]
    return Plan(Buffer, ctypes.cast(symbol, ctypes.c_void_p).value, parameters, (0, 1, 2), 3), calls, symbol


def test_plan_passes_addresses_and_extents(plan_and_calls):
    from weft_b200.runtime import Buffer

    plan, calls, _ = plan_and_calls
    w = Buffer(np.zeros(4 * 288, np.uint8), shape=(4, 512), encoding="Q4_K")
    x, y = Buffer(np.zeros((2, 512), np.float32)), Buffer(np.zeros((2, 4), np.float32))
    xq = Buffer(np.zeros(2 * 584, np.uint8), shape=(2, 512), encoding="Q8_K")
    assert plan(w, x, xq, y) == 0
    assert calls[-1] == (w.address, x.address, xq.address, y.address, 4, 512, 2)
    y.shape = (2, 5)                       # fields are read at each call
    assert plan(w, x, xq, y) is None


@pytest.mark.parametrize("change", ["type", "encoding", "rank", "extent", "records", "short", "alignment", "readonly", "alias", "count", "keyword"])
def test_plan_leaves_what_it_cannot_vouch_for(plan_and_calls, change):
    from weft_b200.runtime import Buffer

    plan, calls, _ = plan_and_calls
    shared = np.zeros(2 * 584 + 64, np.uint8)
    w = Buffer(np.zeros(4 * 288, np.uint8), shape=(4, 512), encoding="Q4_K")
    x, y = Buffer(np.zeros((2, 512), np.float32)), Buffer(np.zeros((2, 4), np.float32))
    xq = Buffer(shared[:2 * 584], shape=(2, 512), encoding="Q8_K")
    args, kwargs = [w, x, xq, y], {}
    if change == "type": args[1] = np.zeros((2, 512), np.float32)
    if change == "encoding": args[2] = Buffer(np.zeros(2 * 584, np.uint8), shape=(2, 512), encoding="Q8_0")
    if change == "rank": args[3] = Buffer(np.zeros(8, np.float32))
    if change == "extent": args[3] = Buffer(np.zeros((3, 4), np.float32))
    if change == "records": args[0], args[1] = Buffer(np.zeros(4 * 288, np.uint8), shape=(4, 500), encoding="Q4_K"), Buffer(np.zeros((2, 500), np.float32))
    if change == "short": args[0] = Buffer(np.zeros(100, np.uint8), shape=(4, 512), encoding="Q4_K")
    if change == "alignment": args[2] = Buffer(shared[2:2 + 2 * 584], shape=(2, 512), encoding="Q8_K")
    if change == "readonly": args[3] = Buffer(bytes(32), shape=(2, 4), encoding="dense.f32")
    if change == "alias": args[3] = Buffer(shared[:32].view(np.float32), shape=(2, 4))
    if change == "count": args = args[:3]
    if change == "keyword": kwargs = {"N": 4}
    before = len(calls)
    assert plan(*args, **kwargs) is None
    assert len(calls) == before
