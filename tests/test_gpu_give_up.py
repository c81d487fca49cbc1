"""Roles of the tcgen05 kernels for batches that give up: the call ends with a status, and the next one is not affected.

With TileArgs::most_blocks below what a CTA needs its record warp gives up, and all others wait for records that nobody fetches.  Copies, MMAs
and arrivals are under way then: they have to be waited for before the CTA leaves, since the next one on the SM gets the same shared and
tensor memory.
"""
from __future__ import annotations

import ctypes

import pytest

from test_dispatch_bounds import TileArgs, library
from test_gpu_batch import Problem, lib, torch  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu

WAIT_RAN_OUT = 1


@pytest.fixture(scope="module")
def kernels():
    built = library()
    pair, fold = built["_ZN4weft11launch_pairERKNS_8TileArgsEPhPiiP11CUstream_stPj"], built["_ZN4weft11launch_foldERKNS_8TileArgsEPhPiiP11CUstream_stPj"]
    pair_bytes, fold_bytes = built["_ZN4weft16pair_plane_bytesERKNS_8TileArgsEi"], built["_ZN4weft16fold_plane_bytesERKNS_8TileArgsE"]
    for launch in (pair, fold):
        launch.argtypes = [ctypes.POINTER(TileArgs), ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.POINTER(ctypes.c_uint)]
    pair_bytes.restype = fold_bytes.restype = ctypes.c_size_t
    return {"pairs": (pair, lambda args, sms: pair_bytes(ctypes.byref(args), sms)), "fold": (fold, lambda args, sms: fold_bytes(ctypes.byref(args)))}


@pytest.mark.parametrize("blocks", [0, 1, 2])
@pytest.mark.parametrize("kernel, name, mnk", [("pairs", "Q4_K", (300, 2311, 4096)), ("pairs", "Q5_K", (129, 2311, 4096)), ("pairs", "Q6_K", (129, 2311, 4096)),
                                               ("pairs", "TQ1_0", (257, 9371, 1280)), ("pairs", "Q4_0", (128, 3001, 4352)), ("pairs", "Q8_0", (255, 9371, 1280)),
                                               ("pairs", "Q6_K", (700, 19331, 1024)), ("fold", "Q4_K", (33, 4099, 4096)), ("fold", "Q4_K", (100, 19000, 2048))])
def test_a_role_that_gives_up(torch, lib, oracle, golden, kernels, kernel, name, mnk, blocks):  # noqa: F811
    problem, (launch, plane_bytes) = Problem(torch, oracle, golden, name, *mnk), kernels[kernel]
    sms, launches = torch.cuda.get_device_properties(0).multi_processor_count, ctypes.c_uint()
    args = TileArgs(problem.fmt, problem.w.data_ptr(), problem.x.data_ptr(), problem.xq.data_ptr(), None, None, problem.powers.data_ptr(), problem.y.data_ptr(),
                    problem.n, problem.k, problem.m, problem.n, blocks)
    planes, status = torch.empty(plane_bytes(args, sms), dtype=torch.uint8, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    for _ in range(5):
        args.most_blocks = blocks
        status.zero_()
        assert launch(ctypes.byref(args), planes.data_ptr(), status.data_ptr(), sms, stream, ctypes.byref(launches)) == 0
        assert int(status) == WAIT_RAN_OUT
        args.most_blocks = 2 ** 31 - 1             # the CTAs that follow find shared and tensor memory free and unwritten
        problem.y.fill_(float("nan"))
        status.zero_()
        assert launch(ctypes.byref(args), planes.data_ptr(), status.data_ptr(), sms, stream, ctypes.byref(launches)) == 0
        assert int(status) == 0
        problem.check()
