"""GPU parity of the contractions with the weights in tensor memory against the CPU oracle: fold_kernel on every size with Q4_K, and what the
dispatch takes for the formats that have CTA pairs (test_gpu_pairs.py has the edges of those).

Sizes sit at the edges of fold_kernel's tiles: rows that do not fill the last 128, a matrix of eight rows, tokens just above a tile, one block
of K, blocks that do not divide among the slices of K, more tiles than SMs, a last round of few rows that is a launch of its own.

Bound: 1e-5 relative L2 and the reference harnesses' |a - e| <= 1e-4 + 2e-3 |e|.  The sums of a block are integers, held
exactly by the accumulators; the block's sum is rounded once (Q4_K: in its last accumulation step, by at most 2^-23).
"""
from __future__ import annotations

import numpy as np
import pytest

from direct import run_on
from helpers import rel_l2
from test_gpu_batch import Problem, lib, torch  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu

FORMATS = ["Q4_K", "Q5_K", "Q6_K"]


def check_both_sources(torch, lib, problem, kernel=None):  # noqa: F811
    """With X and with the caller's records instead: the same planes, the same bits.  kernel: this one, not the dispatch's choice."""
    def run(flags):
        problem.y.fill_(float("nan"))
        torch.cuda.synchronize()
        if kernel is None:
            problem.run(lib, flags)
        else:
            assert run_on(kernel, torch, problem, flags)[0] == 0

    run(0)
    problem.check()
    first = problem.y.clone()
    run(1)
    assert torch.equal(problem.y, first)


def check_all(torch, lib, problem, name):  # noqa: F811
    check_both_sources(torch, lib, problem)
    if name == "Q4_K":
        check_both_sources(torch, lib, problem, "fold")


@pytest.mark.parametrize("name", FORMATS)
@pytest.mark.parametrize("mnk", [(33, 4099, 4096), (129, 1027, 4352), (300, 8, 229632), (700, 3105, 256), (58, 18949, 512), (33, 18957, 4096)])
def test_tile_edges(torch, lib, oracle, golden, name, mnk):  # noqa: F811
    check_all(torch, lib, Problem(torch, oracle, golden, name, *mnk), name)


@pytest.mark.parametrize("name", FORMATS)
@pytest.mark.parametrize("mnk", [(65, 5643, 4096), (129, 2707, 4352), (300, 24, 229632), (700, 8377, 256), (90, 32571, 512), (97, 3779, 4096), (66, 18957, 4096)])
def test_tile_edges_further_on(torch, lib, oracle, golden, name, mnk):  # noqa: F811
    check_all(torch, lib, Problem(torch, oracle, golden, name, *mnk), name)


@pytest.mark.parametrize("name", ["Q4_K", "Q6_K"])
@pytest.mark.parametrize("mnk", [(33, 6689, 4096), (48, 4587, 4096), (300, 16, 229632)])
def test_narrow_tiles(torch, lib, oracle, golden, name, mnk):  # noqa: F811
    check_all(torch, lib, Problem(torch, oracle, golden, name, *mnk), name)


@pytest.mark.parametrize("name", ["Q4_K", "Q5_K"])
def test_fewest_tokens(torch, lib, oracle, golden, name):  # noqa: F811
    check_all(torch, lib, Problem(torch, oracle, golden, name, 25, 3190, 15360), name)


@pytest.mark.parametrize("mnk, launches", [((32, 18945, 4096), 3), ((32, 18951, 4096), 3), ((30, 18957, 4096), 3),      # a second launch of 1, 7 and 13 rows
                                           ((28, 9473, 6912), 2), ((30, 40001, 1280), 2)])                            # K in one slice: a tile a CTA, and several
def test_one_slice_and_second_launches(torch, lib, oracle, golden, mnk, launches):  # noqa: F811
    problem = Problem(torch, oracle, golden, "Q4_K", *mnk)
    assert run_on("fold", torch, problem) == (0, launches)
    check_both_sources(torch, lib, problem, "fold")
    check_both_sources(torch, lib, problem)


def check_kernels(torch, lib, problem, name, flags=0):  # noqa: F811
    """The dispatch's choice, CTA pairs, and fold_kernel where it has the format."""
    problem.run(lib, flags)
    problem.check()
    for kernel in ["pairs", "fold"][:2 if name == "Q4_K" else 1]:
        problem.y.fill_(float("nan"))
        assert run_on(kernel, torch, problem, flags)[0] == 0
        problem.check()


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
    check_kernels(torch, lib, Problem(torch, oracle, golden, name, 66, 5700, 4096), name)


class Records(Problem):
    """A problem whose weights and activation records are given: codes (m, k), every scale of the activations 1."""

    def __init__(self, torch, oracle, name, w, codes, n):  # noqa: F811
        self.fmt, (self.m, self.k), self.n = oracle.FORMAT_IDS[name], codes.shape, n
        blocks = codes.reshape(self.m, -1, 256)
        records = np.zeros((self.m, blocks.shape[1], 292), np.uint8)
        records[:, :, :4] = np.float32(1).reshape(1).view(np.uint8)
        records[:, :, 4:260] = blocks.view(np.uint8)
        records[:, :, 260:] = blocks.reshape(self.m, -1, 16, 16).sum(-1, dtype=np.int16).view(np.uint8).reshape(self.m, -1, 32)
        self.want_xq = records.reshape(self.m, -1)
        self.want, _ = oracle.mul_mat(self.fmt, w, None, n, self.k, self.m, xq=self.want_xq)
        self.w, self.xq = torch.from_numpy(w).cuda(), torch.from_numpy(self.want_xq).cuda()
        self.grid = self.signs = self.powers = self.x = self.xq
        self.y = torch.full((self.m, n), float("nan"), device="cuda")


RECORD_BYTES, ONE = {"Q4_K": 144, "Q5_K": 176, "Q6_K": 210}, np.float16(1).reshape(1).view(np.uint8)


@pytest.mark.parametrize("name", FORMATS)
@pytest.mark.parametrize("m", [66, 90, 128])
def test_large_partial_sums_that_cancel(torch, lib, oracle, name, m):  # noqa: F811
    """Largest weights against activations of one sign, then of the other: the sum of a block passes 2^24 and comes back to a few
    thousand.  The integer sums are exact, so the bound is the one of the additions over 16 blocks."""
    rng = np.random.default_rng(m)
    n, k = 5700, 4096
    w = np.full((n, k // 256, RECORD_BYTES[name]), 0xFF, np.uint8)
    if name == "Q6_K":
        w[:, :, 192:208], w[:, :, 208:] = 0x7F, ONE
    else:
        w[:, :, :2], w[:, :, 2:4] = ONE, 0
    codes = np.full((m, k // 256, 256), 127, np.int8)
    codes[:, :, 128:] = -127
    codes[:, :, 128:136] += rng.integers(0, 3, size=(m, k // 256, 8), dtype=np.int8)
    check_kernels(torch, lib, Records(torch, oracle, name, w.reshape(n, -1), codes.reshape(m, k), n), name, flags=1)
    if name != "Q6_K":                               # the first 160 of a block against its last 96
        first = np.arange(k) % 256 < 160
        codes = np.where(first, 127 - rng.integers(0, 2, size=(m, k)), -127).astype(np.int8)
        check_kernels(torch, lib, Records(torch, oracle, name, w.reshape(n, -1), codes, n), name, flags=1)


@pytest.mark.parametrize("name", FORMATS)
@pytest.mark.parametrize("m", [66, 90, 128, 700])
def test_integer_sums_are_exact(torch, lib, oracle, name, m):  # noqa: F811
    """One block, every bit of codes, scales and mins random, all super-scales 1: the results are integers."""
    rng = np.random.default_rng(m)
    n, k = int(1.5e9 / m / 256) // 128 * 128 + 131, 256
    w = rng.integers(0, 256, size=(n, RECORD_BYTES[name]), dtype=np.uint8)
    if name == "Q6_K": w[:, 208:] = ONE
    else: w[:, :2], w[:, 2:4] = ONE, ONE
    codes = rng.integers(-127, 128, size=(m, k), dtype=np.int8)
    codes[m // 2:] = np.abs(codes[m // 2:])          # large sums of one sign
    problem = Records(torch, oracle, name, w, codes, n)
    whole = np.abs(problem.want) < 2.0 ** 24
    for kernel in [None, "pairs", "fold"][:3 if name == "Q4_K" else 2]:
        problem.y.fill_(float("nan"))
        torch.cuda.synchronize()
        if kernel is None:
            problem.run(lib, flags=1)
        else:
            assert run_on(kernel, torch, problem, flags=1)[0] == 0
        got = problem.y.cpu().numpy()
        assert np.array_equal(got[whole], problem.want[whole]), kernel
        assert rel_l2(got, problem.want) <= 2.0 ** -23, kernel
