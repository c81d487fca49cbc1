"""Roles of the tcgen05 kernels for batches that give up: the call ends with a status, and the next one is not affected.

With TileArgs::most_blocks below what a CTA needs its record warp gives up, and all others wait for records that nobody fetches.  Copies, MMAs
and arrivals are under way then: they have to be waited for before the CTA leaves, since the next one on the SM gets the same shared and
tensor memory.
"""
from __future__ import annotations

import pytest

from direct import run_on
from test_gpu_batch import Problem, torch  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu

WAIT_RAN_OUT = 1


@pytest.mark.parametrize("blocks", [0, 1, 2])
@pytest.mark.parametrize("kernel, name, mnk", [("pairs", "Q4_K", (300, 2311, 4096)), ("pairs", "Q5_K", (129, 2311, 4096)), ("pairs", "Q6_K", (129, 2311, 4096)),
                                               ("pairs", "TQ1_0", (257, 9371, 1280)), ("pairs", "Q4_0", (128, 3001, 4352)), ("pairs", "Q8_0", (255, 9371, 1280)),
                                               ("pairs", "Q6_K", (700, 19331, 1024)), ("fold", "Q4_K", (33, 4099, 4096)), ("fold", "Q4_K", (100, 19000, 2048))])
def test_a_role_that_gives_up(torch, oracle, golden, kernel, name, mnk, blocks):  # noqa: F811
    problem = Problem(torch, oracle, golden, name, *mnk)
    for _ in range(5):
        assert run_on(kernel, torch, problem, most_blocks=blocks)[0] == WAIT_RAN_OUT
        problem.y.fill_(float("nan"))
        assert run_on(kernel, torch, problem)[0] == 0        # the CTAs that follow find shared and tensor memory free and unwritten
        problem.check()
