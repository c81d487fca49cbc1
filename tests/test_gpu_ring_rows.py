"""Decode products of matrices whose rows are no multiple of 16 bytes (the ring kernel starts its copies before them and moves
the last few bytes itself) against the CPU oracle: one to eight records in all (every remainder of the matrix's last 16 bytes),
a stage per CTA and less, several stages with a ragged tail, rows longer than a stage.  Bound as for the other decode products:
the integer sums are exact, only the order of the fp32 additions differs (1e-5 relative L2).
"""
from __future__ import annotations

import pytest

import test_gpu_parity as parity
from test_gpu_parity import torch, weft  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu

FORMATS = ["q2_k", "q3_k", "q6_k", "iq2_xxs", "tq1_0", "iq2_xs", "iq3_xxs", "iq2_s", "iq3_s", "iq1_s", "iq1_m"]


@pytest.mark.parametrize("name", FORMATS)
@pytest.mark.parametrize("shape", [(n, 256) for n in range(1, 9)] + [(7, 768), (1193, 2816), (9001, 1280), (301, 14080)])
def test_rows_at_any_even_address(torch, weft, oracle, golden, name, shape):  # noqa: F811
    parity.test_vec_dot_rows_against_oracle(torch, weft, oracle, golden, name, shape)


@pytest.mark.parametrize("name", [name for name in FORMATS if name in parity.DECODE_FORMATS])
@pytest.mark.parametrize("mnk", [(1, 3, 256), (2, 1193, 2816)])
def test_quantizing_launch(torch, weft, oracle, golden, name, mnk):  # noqa: F811
    parity.test_mul_mat_decode(torch, weft, oracle, golden, name, mnk)


@pytest.mark.parametrize("mnk", [(1, 1, 256), (1, 5, 1024), (1, 301, 2048), (1, 300, 2304), (2, 149, 4352), (1, 3001, 6144), (1, 301, 6400)])
def test_q4_k_rows_by_half_warps(torch, weft, oracle, golden, mnk):  # noqa: F811
    """Up to 16 half-records of a row left after whole passes of 32 go to half a warp per row: K at both sides of the line."""
    parity.test_mul_mat_decode(torch, weft, oracle, golden, "q4_k", mnk)
