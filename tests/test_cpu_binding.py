"""The Python binding's calls with declared argument types refuse what the others refuse."""
import ctypes as C

import numpy as np
import pytest
import torch

from flagcx_b200 import capi


def test_arguments_that_are_no_numbers_or_buffers_are_refused():
    nobody = capi.Comm(C.c_void_p(0), owns=False)
    x = np.zeros(4, dtype=np.float32)
    for buf in (x, torch.zeros(4), x.ctypes.data, None):
        with pytest.raises(capi.FlagcxError):  # the library's answer: no communicator
            nobody.all_reduce(buf, buf, 4, capi.FLOAT)
    for count in (1.5, "4", None):
        with pytest.raises(TypeError):
            nobody.all_reduce(x, x, count, capi.FLOAT)
    for buf in ([0.0], "x", object()):
        with pytest.raises(TypeError):
            nobody.all_reduce(buf, x, 4, capi.FLOAT)
    with pytest.raises(TypeError):
        nobody.all_reduce(x, x, 4, capi.FLOAT, stream="default")


def test_gemm_refuses_tensors_of_the_host():
    from flagcx_b200.parallel.tp import gemm_bf16
    a = torch.zeros(128, 64, dtype=torch.bfloat16)
    with pytest.raises((ValueError, RuntimeError, AssertionError)):  # torch has no current stream for them
        gemm_bf16(a, torch.zeros(256, 64, dtype=torch.bfloat16))
