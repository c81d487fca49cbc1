"""GPU parity of the contraction with the weights in tensor memory (larger batches of Q4_K, Q5_K, Q6_K) against the CPU oracle.

Sizes are the smallest that reach it (above 32 tokens and 5.5e8 products; Q4_K and Q5_K from 25 tokens and 1.2e9) and sit at
the edges of its tiles: rows that do not fill the last 128 (nor, for Q6_K, the last super-row of 8), a matrix of eight rows,
tokens just above a tile, one block of K, blocks that do not divide among the slices of K, more tiles than SMs, a last round of
13 rows that is a launch of its own.

Bound: 1e-5 relative L2 and the reference harnesses' |a - e| <= 1e-4 + 2e-3 |e|.  The sums of a block are integers in fp32
accumulators, exact below 2^24; above, the 16 accumulation steps of a block (Q6_K: 32, two operands) each lose at most
2^-23 of the running sum, so terms of one sign lose at most 32 * 2^-23 = 3.9e-6.
"""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_batch import Problem, lib, torch  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu

FORMATS = ["Q4_K", "Q5_K", "Q6_K"]


def check_both_sources(torch, lib, problem):  # noqa: F811
    problem.run(lib)
    problem.check()
    first = problem.y.clone()                      # the caller's records instead of X: the same planes, the same bits
    problem.y.fill_(float("nan"))
    torch.cuda.synchronize()
    problem.run(lib, flags=1)
    assert torch.equal(problem.y, first)


@pytest.mark.parametrize("name", FORMATS)
@pytest.mark.parametrize("mnk", [(33, 4099, 4096), (129, 1027, 4352), (300, 8, 229632), (700, 3105, 256), (58, 18949, 512), (33, 18957, 4096)])
def test_tile_edges(torch, lib, oracle, golden, name, mnk):  # noqa: F811
    check_both_sources(torch, lib, Problem(torch, oracle, golden, name, *mnk))


@pytest.mark.parametrize("name", ["Q4_K", "Q5_K"])
def test_fewest_tokens(torch, lib, oracle, golden, name):  # noqa: F811
    check_both_sources(torch, lib, Problem(torch, oracle, golden, name, 25, 3190, 15360))


@pytest.mark.parametrize("name", FORMATS)
def test_largest_codes_and_scales(torch, lib, oracle, golden, name, monkeypatch):  # noqa: F811
    """Every weight and every scale at its largest, all activations alike: the sums go past 2^24."""
    import test_gpu_batch as batch

    def largest(fmt, rng, n, k):
        w = draw_weights(fmt, rng, n, k)
        records = w.reshape(-1, 210 if name == "Q6_K" else {"Q4_K": 144, "Q5_K": 176}[name])
        if name == "Q6_K":
            records[:, :192], records[:, 192:208] = 0xFF, 0x7F
        else:
            records[:, 4:] = 0xFF
        return w

    draw_weights = batch.weights
    monkeypatch.setattr(batch, "weights", largest)
    monkeypatch.setattr(batch, "activations", lambda rng, m, k: np.full((m, k), 0.75, dtype=np.float32))
    problem = Problem(torch, oracle, golden, name, 64, 2200, 4096)
    problem.run(lib)
    problem.check()
