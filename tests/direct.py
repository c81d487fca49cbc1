"""Launches of a batch kernel whatever the dispatch would choose (test infrastructure)."""
from __future__ import annotations

import ctypes
import functools

from test_dispatch_bounds import TileArgs, library

ALL_BLOCKS = 2 ** 31 - 1


@functools.lru_cache(maxsize=None)
def _entry(kernel: str):
    built = library()
    launch = built["_ZN4weft11launch_%sERKNS_8TileArgsEPhPiiP11CUstream_stPj" % {"pairs": "pair", "fold": "fold"}[kernel]]
    launch.argtypes = [ctypes.POINTER(TileArgs), ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.POINTER(ctypes.c_uint)]
    plane_bytes = built["_ZN4weft16pair_plane_bytesERKNS_8TileArgsEi" if kernel == "pairs" else "_ZN4weft16fold_plane_bytesERKNS_8TileArgsE"]
    plane_bytes.restype = ctypes.c_size_t
    return launch, plane_bytes


def run_on(kernel: str, torch, problem, flags: int = 0, most_blocks: int = ALL_BLOCKS) -> tuple[int, int]:
    """The kernel ("pairs" or "fold") on a problem of test_gpu_batch; its device status and how many launches it took."""
    launch, plane_bytes = _entry(kernel)
    args = TileArgs(problem.fmt, problem.w.data_ptr(), None if flags else problem.x.data_ptr(), problem.xq.data_ptr(), None, None, problem.powers.data_ptr(),
                    problem.y.data_ptr(), problem.n, problem.k, problem.m, problem.n, most_blocks)
    sms, launches = torch.cuda.get_device_properties(0).multi_processor_count, ctypes.c_uint()
    planes = torch.empty(plane_bytes(ctypes.byref(args), sms) if kernel == "pairs" else plane_bytes(ctypes.byref(args)), dtype=torch.uint8, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    assert launch(ctypes.byref(args), planes.data_ptr(), status.data_ptr(), sms, stream, ctypes.byref(launches)) == 0
    return int(status), launches.value
