"""Arguments that a gather launcher cannot serve are refused, on the host."""
import ctypes
import os

import pytest

LIB = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "claire_b200", "libclaire_b200.so")
INVALID_VALUE = 1  # cudaErrorInvalidValue


class Dims(ctypes.Structure):
    _fields_ = [("n1", ctypes.c_int), ("n2", ctypes.c_int), ("n3", ctypes.c_int)]


# cb::launch_interp16(const bf16*, long long, const float*, long long, const int4*, long long, bf16*, long long,
#                     int, const Dims&, const int*, cudaStream_t)
INTERP16 = "_ZN2cb15launch_interp16EPK13__nv_bfloat16xPKfxPK4int4xPS0_xiRKNS_4DimsEPKiP11CUstream_st"


@pytest.mark.parametrize("nprob,masked", [(2, False), (1, True), (3, True)])
def test_bf16_gather_without_a_table_takes_one_unmasked_problem(nprob, masked):
    """The kernel without a table gathers problem 0 and reads no mask: a batch
    or a mask must not be dropped in silence."""
    p, ll = ctypes.c_void_p, ctypes.c_longlong
    fn = getattr(ctypes.CDLL(LIB), INTERP16)
    fn.restype = ctypes.c_int
    # host memory that stands for device arrays: nothing may be launched on it
    d, n = Dims(16, 16, 16), 16 ** 3
    f, disp, out = ((ctypes.c_float * (3 * 3 * n))() for _ in range(3))
    mask = (ctypes.c_int * nprob)(*[1] * nprob)
    rc = fn(ctypes.byref(f), ll(n), ctypes.byref(disp), ll(3 * n), p(None), ll(0), ctypes.byref(out), ll(n),
            ctypes.c_int(nprob), ctypes.byref(d), ctypes.byref(mask) if masked else p(None), p(None))
    assert rc == INVALID_VALUE
