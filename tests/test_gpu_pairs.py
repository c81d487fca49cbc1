"""GPU parity of the contraction on CTA pairs (larger batches of Q4_K, Q5_K, Q6_K, TQ1_0, Q4_0 and Q8_0) against the CPU oracle.

The kernel is launched whatever the dispatch would choose for a size; sizes sit at the edges of its tiles: rows
that do not fill the last 256, nor the last super-row of 8, a matrix of eight rows, tokens just above a chunk and a tile, one block of K,
fewer tiles than pairs (each shared by several, or all shared by all pairs so that runs span two tiles), more tiles than pairs with the rest
whole or shared.

Bound: 1e-5 relative L2 and the reference harnesses' |a - e| <= 1e-4 + 2e-3 |e|: the sums of a block are integers and exact, only the
order of the fp32 additions over the blocks differs.
"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from direct import run_on
from helpers import rel_l2
from test_gpu_batch import Problem, lib, torch  # noqa: F401  (fixtures)
from test_gpu_fold import check_both_sources
from test_dispatch_bounds import pair_supported  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

FORMATS, GROUPED = ["Q4_K", "Q5_K", "Q6_K", "TQ1_0"], ["Q4_0", "Q8_0"]


@pytest.mark.parametrize("name", FORMATS)
@pytest.mark.parametrize("mnk", [(129, 2311, 4096),          # few tiles, each shared by several pairs
                                 (300, 8, 512000),           # one row tile of eight rows, two thousand blocks
                                 (257, 9371, 512),           # a second tile of one token
                                 (700, 6703, 256),           # one block: nothing to share
                                 (40, 14341, 2304),          # one chunk; fewer tiles than pairs, blocks that do not divide
                                 (40, 14341, 4096),
                                 (300, 1283, 14336),         # fewer tiles than pairs, shared by all of them
                                 (65, 19331, 1024),          # more tiles than pairs
                                 (512, 5003, 768)])
def test_tile_edges(torch, lib, oracle, golden, name, mnk):  # noqa: F811
    check_both_sources(torch, lib, Problem(torch, oracle, golden, name, *mnk), "pairs")


@pytest.mark.parametrize("name", ["Q6_K", "TQ1_0"])            # records at any even address
@pytest.mark.parametrize("n", [3081, 3210, 3083, 3212, 3085, 3214, 3087])
def test_rows_after_the_last_super_row(torch, lib, oracle, golden, name, n):  # noqa: F811
    """One to seven rows, in the even and in the odd CTA of a pair; the last record ends at every offset from a 16-byte boundary that there is."""
    check_both_sources(torch, lib, Problem(torch, oracle, golden, name, 310, n, 1280), "pairs")


@pytest.mark.parametrize("name", GROUPED)                      # tiles of 128 tokens, a scale pair per 32 elements
@pytest.mark.parametrize("mnk", [(128, 3001, 4352),          # few tiles, each shared by several pairs
                                 (500, 2311, 2304),          # fewer tiles than pairs, blocks that do not divide
                                 (250, 6703, 1280),          # a tile each, some pairs idle
                                 (255, 9371, 768),           # a tile for each of 74 pairs
                                 (384, 19331, 256),          # one block: nothing to share
                                 (640, 9001, 1024)])         # more tiles than pairs, the rest shared
def test_group_tile_edges(torch, lib, oracle, golden, name, mnk):  # noqa: F811
    check_both_sources(torch, lib, Problem(torch, oracle, golden, name, *mnk), "pairs")


@pytest.mark.parametrize("m, n, k", [(130, 2311, 4096), (300, 8203, 512)])
def test_infinite_scales_of_ternary_records(torch, lib, oracle, golden, m, n, k, monkeypatch):  # noqa: F811
    """Records whose f16 scale is infinite or NaN: what the oracle gives, infinities with their signs."""
    import test_gpu_batch as batch

    def overflown(fmt, rng, n, k):
        w = draw_weights(fmt, rng, n, k)
        d = w.reshape(n, k // 256, 54)[:, :, 52:]
        d[5, 0], d[70, -1], d[n - 1, 0], d[n - 9, 1] = [0, 0x7c], [0, 0xfc], [0, 0x7c], [0, 0x7e]
        return w

    draw_weights = batch.weights
    monkeypatch.setattr(batch, "weights", overflown)
    problem = Problem(torch, oracle, golden, "TQ1_0", m, n, k)
    assert run_on("pairs", torch, problem)[0] == 0
    got, rows = problem.y.cpu().numpy(), [5, 70, n - 9, n - 1]
    assert np.isinf(problem.want[:, rows[:2]]).any() and np.isnan(problem.want[:, n - 9]).all()
    assert np.array_equal(got[:, rows], problem.want[:, rows], equal_nan=True)
    assert rel_l2(np.delete(got, rows, axis=1), np.delete(problem.want, rows, axis=1)) <= 1e-5


@pytest.mark.parametrize("name", GROUPED)
def test_infinite_scales_of_groups(torch, lib, oracle, golden, name, monkeypatch):  # noqa: F811
    """Records of 32 elements whose f16 scale is infinite or NaN: the rows are what the oracle gives, NaN where its sums are."""
    import test_gpu_batch as batch

    def overflown(fmt, rng, n, k):
        w = draw_weights(fmt, rng, n, k)
        d = w.reshape(n, k // 32, -1)[:, :, :2]
        d[5, 0], d[70, -1], d[n - 1, 3], d[n - 9, 1] = [0, 0x7c], [0, 0xfc], [0, 0x7c], [0, 0x7e]
        return w

    draw_weights = batch.weights
    monkeypatch.setattr(batch, "weights", overflown)
    problem = Problem(torch, oracle, golden, name, 250, 2311, 4096)
    assert run_on("pairs", torch, problem)[0] == 0
    got, rows = problem.y.cpu().numpy(), [5, 70, 2311 - 9, 2311 - 1]
    assert np.isinf(problem.want[:, rows[:2]]).any() and np.isnan(problem.want[:, 2311 - 9]).all()
    assert np.array_equal(got[:, rows], problem.want[:, rows], equal_nan=True)
    assert rel_l2(np.delete(got, rows, axis=1), np.delete(problem.want, rows, axis=1)) <= 1e-5


@pytest.mark.parametrize("name, mnk, kernels", [("Q6_K", (700, 6703, 256), 2),      # one block of K: more tiles than pairs, nothing to share
                                                ("Q8_0", (384, 19331, 256), 2),
                                                ("Q5_K", (512, 5003, 768), 2),
                                                ("TQ1_0", (129, 2311, 4096), 3)])
def test_launches_are_counted_as_they_are_made(torch, lib, oracle, golden, name, mnk, kernels):  # noqa: F811
    """Planes, contraction and, where tiles are shared, the kernel that adds their parts: as many as a capture of the call holds."""
    problem, graph, side = Problem(torch, oracle, golden, name, *mnk), torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
    nodes = ctypes.c_size_t()
    lib.weft_b200_set_async(1)
    lib.weft_b200_set_stream(ctypes.c_void_p(side.cuda_stream))
    try:
        before = lib.weft_b200_launch_count()
        with torch.cuda.graph(graph, stream=side):
            problem.run(lib)
        counted = lib.weft_b200_launch_count() - before
        assert ctypes.CDLL("libcuda.so.1").cuGraphGetNodes(ctypes.c_void_p(graph.raw_cuda_graph()), None, ctypes.byref(nodes)) == 0
    finally:
        lib.weft_b200_set_stream(None)
        lib.weft_b200_set_async(0)
    assert (nodes.value, counted) == (kernels, kernels)


@pytest.mark.parametrize("m, n, k, pairs", [(68, 8416, 6912, False), (380, 6158, 4864, False), (122, 8841, 6912, False), (512, 14336, 4096, True), (512, 4096, 14336, True),
                                            (160, 4096, 4096, True), (77, 28672, 8192, True)])
def test_pairs_and_single_ctas_by_what_was_measured(torch, lib, pair_supported, m, n, k, pairs):  # noqa: F811
    """Q4_K at sizes where one of the two is quicker by 5 % and more.  How many clusters the device holds decides with."""
    assert pair_supported(8, m, n, k, sms=torch.cuda.get_device_properties(0).multi_processor_count) == pairs


@pytest.mark.parametrize("m, n, k", [((1 << 20) + 3, 13, 2048), ((1 << 20) + 130, 5, 2048), (129, 9, (1 << 22) + 2048)])
def test_ternary_batches_of_any_extent(torch, lib, oracle, golden, m, n, k):  # noqa: F811
    """More than 2^20 tokens, fewer than eight rows of them, and rows of more than 2^22 elements: a few distinct tokens, repeated."""
    few = Problem(torch, oracle, golden, "TQ1_0", 257 if m > 257 else 3, n, k)
    times = -(-m // few.m)
    x, xq, y = few.x.repeat(times, 1)[:m].contiguous(), torch.zeros((m, few.xq.shape[1]), dtype=torch.uint8, device="cuda"), torch.full((m, n), float("nan"), device="cuda")
    torch.cuda.synchronize()
    assert lib.weft_b200_mul_mat_shard(few.fmt, 1, few.w.data_ptr(), x.data_ptr(), xq.data_ptr(), None, None, few.powers.data_ptr(), y.data_ptr(), n, k, m, n, 0) == 0
    torch.cuda.synchronize()
    few.y.copy_(y[:few.m])
    few.xq.copy_(xq[:few.m])
    few.check()
    assert torch.equal(xq, few.xq.repeat(times, 1)[:m])
    # tiles that pairs share are added up in parts: up to k / 256 additions that round in another order, by 2^-24 each
    want = few.y.repeat(times, 1)[:m].double()
    assert float((y - want).norm() / want.norm()) <= max(8, k // 256) ** 0.5 * 2.0 ** -24
    assert bool(((y - want).abs() <= 1e-4 + 2e-3 * want.abs()).all())
